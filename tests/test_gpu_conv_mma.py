"""The tensor-core 3x3 convolutions at the edges of their tiles (channel counts around 8, 16, 32 and
128, tiles of 16 and 32 pixels, bases that are not 4-byte aligned, infinities and NaN) against
FP64 convolutions of the same BF16 activations and FP32 weights.

Outputs are BF16: their rounding is at most 2^-9 of each value, 2.5e-3 bounds it and the FP32
sums. The weight gradient adds 128 pixels per accumulation in the tensor core, eight truncating
adds of at most 2^-23 each: 1e-6 of the norm."""
import ctypes

import numpy as np
import pytest

from golden_io import rel_l2

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _bf16(rng, shape, offset, scale=1.0):
    """A BF16 CUDA tensor whose base lies `offset` elements behind a 256-byte boundary."""
    import torch
    n = int(np.prod(shape))
    buf = torch.zeros(n + 8, dtype=torch.bfloat16, device="cuda")
    view = buf[offset:offset + n].view(shape)
    view.copy_(torch.from_numpy(rng.normal(size=shape) * scale))
    return view


def _run(x, w, b, dy):
    import torch
    from pypty_gb300 import _lib
    lib, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    (N, Ci, H, W), Co = x.shape, w.shape[0]
    y, dx = torch.empty_like(dy), torch.empty_like(x)
    gw, gb = torch.empty_like(w), torch.empty_like(b)
    n = ctypes.c_int64(0)
    assert lib.pty_nn_conv3x3_wgrad_workspace_floats(N, Ci, Co, H, W, ctypes.byref(n)) == 0
    ws = torch.full((n.value,), float("nan"), device="cuda")
    assert lib.pty_nn_conv3x3(_p(x), _p(w), _p(b), _p(y), N, Ci, Co, H, W, 0, 0, st) == 0
    assert lib.pty_nn_conv3x3(_p(dy), _p(w), None, _p(dx), N, Co, Ci, H, W, 0, 1, st) == 0
    assert lib.pty_nn_conv3x3_wgrad(_p(dy), _p(x), _p(gw), _p(gb), N, Ci, Co, H, W, _p(ws), st) == 0
    torch.cuda.synchronize()
    return y, dx, gw, gb


def _exact(x, w, b, dy):
    import torch
    x, w, b = (t.detach().cpu().double().requires_grad_(True) for t in (x, w, b))
    y = torch.nn.functional.conv2d(x, w, b, padding=1)
    return (y.detach(), *torch.autograd.grad(y, (x, w, b), dy.cpu().double()))


@pytest.mark.parametrize("N,Ci,Co,H,W,offset", [(1, 1, 1, 32, 32, 0), (2, 7, 9, 32, 64, 0), (1, 16, 32, 96, 32, 1),
                                                (3, 17, 33, 32, 32, 0), (1, 33, 65, 64, 32, 3), (1, 130, 12, 32, 32, 0),
                                                (1, 12, 130, 32, 96, 0), (5, 64, 40, 32, 32, 0)])
def test_convolutions_and_gradients(N, Ci, Co, H, W, offset):
    import torch
    rng = np.random.default_rng(Ci * 131 + Co)
    x, dy = _bf16(rng, (N, Ci, H, W), offset), _bf16(rng, (N, Co, H, W), offset, 0.1)
    w = torch.from_numpy(rng.normal(size=(Co, Ci, 3, 3)) * 0.2).float().cuda()
    b = torch.from_numpy(rng.normal(size=Co)).float().cuda()
    got, ref = _run(x, w, b, dy), _exact(x, w, b, dy)
    for k, tol in ((0, 2.5e-3), (1, 2.5e-3), (2, 1e-6), (3, 1e-6)):
        assert rel_l2(got[k].float().cpu().numpy(), ref[k].numpy()) <= tol, k
    again = _run(x, w, b, dy)
    assert all(torch.equal(a, c) for a, c in zip(got, again))


@pytest.mark.parametrize("what", ["x inf", "x nan", "w inf", "w max"])
def test_non_finite_inputs_reach_the_same_outputs(what):
    import torch
    rng = np.random.default_rng(3)
    x, dy = _bf16(rng, (1, 12, 64, 32), 0), _bf16(rng, (1, 20, 64, 32), 0)
    w = torch.from_numpy(rng.normal(size=(20, 12, 3, 3)) * 0.2).float().cuda()
    b = torch.zeros(20, device="cuda")
    if what[0] == "x":
        x[0, 5, 20, 7] = float(what[2:])
        w[3, 5] = 0.0                               # inf * 0
    elif what == "w inf":
        w[4, 2, 1, 1] = float("-inf")
    else:
        w[4, 2, 1, 1] = torch.finfo(torch.float32).max   # finite in FP32, infinite once rounded to BF16
        x.mul_(0.01)
    y = _run(x, w, b, dy)[0].float().cpu().numpy()
    ref = _exact(x, w, b, dy)[0].float().numpy()
    assert np.array_equal(np.isnan(y), np.isnan(ref)) and np.array_equal(np.isposinf(y), np.isposinf(ref))
    assert np.array_equal(np.isneginf(y), np.isneginf(ref))
    ok = np.isfinite(ref) & (np.abs(ref) < 1e30)
    assert rel_l2(y[ok], ref[ok]) <= 2.5e-3
