"""The band limit's tables and streams: tables prepared by a call on one stream, behind work that is
still queued there, are complete when a call on another stream reads them; calls with masks of their own
on two streams share no buffer; a failed preparation is not kept; tables first asked for inside a capture
are the graph's own and not an eager call's. The delays are bounded waits of a few milliseconds."""
import ctypes

import numpy as np
import pytest

from golden_io import rel_l2

pytestmark = pytest.mark.gpu


def _ref(x, cutoff):
    ny, nx = x.shape[:2]
    fy, fx = np.meshgrid(np.fft.fftfreq(ny), np.fft.fftfreq(nx), indexing="ij")
    mask = (fx ** 2 + fy ** 2 <= (0.5 * float(np.float32(cutoff))) ** 2)[:, :, None]
    return np.fft.ifft2(np.fft.fft2(x.astype(np.complex128), axes=(0, 1)) * mask, axes=(0, 1))


def _input(ny, nx, K):
    rng = np.random.default_rng(ny)
    return (rng.normal(size=(ny, nx, K)) + 1j * rng.normal(size=(ny, nx, K))).astype(np.complex64)


@pytest.mark.parametrize("ny,nx", [(64, 128), (256, 64), (128, 2048)])
def test_second_stream_waits_for_the_tables(ny, nx):
    import torch
    from pypty_gb300 import _lib
    from pypty_gb300.engine import Engine
    from pypty_gb300.optim import fourier_clean_
    x = _input(ny, nx, 3)
    xd = torch.from_numpy(x).cuda()
    outs = [torch.zeros_like(xd) for _ in range(3)]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    for s in (a, b):    # the kernels' code is loaded (which waits for the GPU), and memory is there to hand out
        with torch.cuda.stream(s):
            fourier_clean_(xd, 0.6, 0.0, out=outs[0], engine=Engine())
    n = ctypes.c_size_t(0)
    assert _lib.lib().pty_fourier_clean_workspace_bytes(ny, nx, ctypes.byref(n)) == 0
    torch.cuda.synchronize()
    with torch.cuda.stream(a):   # no tables are left in it
        junk = [torch.full((n.value,), 255, dtype=torch.uint8, device="cuda") for _ in range(8)]
        del junk
    torch.cuda.synchronize()
    eng = Engine()
    with torch.cuda.stream(a):
        torch.cuda._sleep(20_000_000)
        fourier_clean_(xd, 0.6, 0.0, out=outs[0], engine=eng)
    with torch.cuda.stream(b):
        fourier_clean_(xd, 0.6, 0.0, out=outs[1], engine=eng)
        fourier_clean_(xd, 0.6, 0.0, out=outs[2], engine=eng)
    torch.cuda.synchronize()
    for o in outs:
        assert rel_l2(o.cpu().numpy(), _ref(x, 0.6)) <= 1e-6


class _Spy:
    """The library with its preparations recorded, the first one refused on request."""

    def __init__(self, lib, refuse=0):
        self.lib, self.refuse, self.buffers = lib, refuse, []

    def __getattr__(self, name):
        f = getattr(self.lib, name)
        if name != "pty_fourier_clean_prepare":
            return f

        def prepare(*args):
            self.buffers.append(args[5])
            if self.refuse:
                self.refuse -= 1
                return -5
            return f(*args)
        return prepare


def test_masks_of_two_streams_share_no_buffer(monkeypatch):
    import torch
    from pypty_gb300 import _lib
    from pypty_gb300.engine import Engine
    from pypty_gb300.optim import fourier_clean_
    spy = _Spy(_lib.lib())
    monkeypatch.setattr(_lib, "lib", lambda: spy)
    x = torch.from_numpy(_input(64, 64, 2)).cuda()
    eng, outs = Engine(), []
    masks = [torch.zeros((64, 64), device="cuda"), torch.ones((64, 64), device="cuda")]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for s, m in zip(streams, masks):
        with torch.cuda.stream(s):
            torch.cuda._sleep(5_000_000)
            outs.append(fourier_clean_(x, mask=m, engine=eng))
    torch.cuda.synchronize()
    assert len(set(spy.buffers)) == 2
    assert not outs[0].any() and rel_l2(outs[1].cpu().numpy(), x.cpu().numpy()) <= 1e-6


def test_failed_preparation_is_not_kept(monkeypatch):
    import torch
    from pypty_gb300 import _lib
    from pypty_gb300.engine import Engine
    from pypty_gb300.optim import fourier_clean_
    spy = _Spy(_lib.lib(), refuse=1)
    monkeypatch.setattr(_lib, "lib", lambda: spy)
    x = _input(64, 128, 1)
    eng, xd = Engine(), torch.from_numpy(x).cuda()
    with pytest.raises(_lib.PtyError):
        fourier_clean_(xd, 0.5, 0.0, engine=eng)
    out = fourier_clean_(xd, 0.5, 0.0, engine=eng)
    fourier_clean_(xd, 0.5, 0.0, engine=eng)
    assert len(spy.buffers) == 2 and rel_l2(out.cpu().numpy(), _ref(x, 0.5)) <= 1e-6


@pytest.mark.parametrize("warm", [False, True])
def test_capture(warm):
    import torch
    from pypty_gb300.engine import Engine
    from pypty_gb300.optim import fourier_clean_
    x = _input(128, 64, 2)
    eng, xd = Engine(), torch.from_numpy(x).cuda()
    out, eager = torch.zeros_like(xd), torch.zeros_like(xd)
    if warm:
        fourier_clean_(xd, 0.6, 0.0, out=eager, engine=eng)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fourier_clean_(xd, 0.6, 0.0, out=out, engine=eng)
    fourier_clean_(xd, 0.6, 0.0, out=eager, engine=eng)     # before the graph has run
    assert rel_l2(eager.cpu().numpy(), _ref(x, 0.6)) <= 1e-6
    for _ in range(2):
        out.zero_()
        graph.replay()
        assert rel_l2(out.cpu().numpy(), _ref(x, 0.6)) <= 1e-6
