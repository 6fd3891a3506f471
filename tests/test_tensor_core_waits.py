"""Tensor-core kernels wait for their MMAs in loops whose trip count differs by lane, and read, allocate
and release tensor memory by instructions that want the warp's lanes together. So, by the sources: no
load from tensor memory follows a bare wait without something that brings the lanes together between
them, and the helpers that allocate and release do so themselves. And a wait that ran out in any thread
marks everything that a weight-gradient block hands out."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pypty_gb300", "csrc")
TOGETHER = ("wait_mma(", "__syncwarp(", "__syncthreads")


def _code(name):
    with open(os.path.join(SRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", ["conv_mma.cuh", "dft_gemm.cu"])
def test_loads_after_a_wait_find_the_warp_together(name):
    code = _code(name)
    tokens = re.findall(r"\bmbar_wait\(|\btmem_ld\w*\(|" + "|".join(re.escape(t) for t in TOGETHER), code)
    assert any(t.startswith("tmem_ld") for t in tokens)
    together = True
    for t in tokens:
        if t == "mbar_wait(":
            together = False
        elif t.startswith("tmem_ld"):
            assert together, "a load from tensor memory after a bare wait"
        else:
            together = True


@pytest.mark.parametrize("name", ["wait_mma", "tmem_alloc", "tmem_dealloc"])
def test_helpers_bring_the_warp_together(name):
    body = re.search(r"void %s\([^)]*\) \{(.*?)\n\}" % name, _code("umma.cuh"), re.S)
    assert body and "__syncwarp();" in body.group(1)
    first = re.search(r"__syncwarp\(\)|asm volatile|fence_after_sync", body.group(1)).group(0)
    assert first == "__syncwarp()"


def test_a_failed_wait_marks_the_whole_share():
    code = _code("conv_mma.cuh")
    kernel = code[code.index("conv3x3_wgrad_mma_kernel("):code.index("strided_sum(")]
    assert re.search(r"failed = __syncthreads_or\(err\)", kernel)
    stores = re.findall(r"(?:pw|pbias)\[[^;]*;", kernel)
    assert len(stores) == 2 and all("failed ? NAN" in s for s in stores)
