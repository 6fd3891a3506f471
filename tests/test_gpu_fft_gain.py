"""The window FFTs and the full-array transforms neither gain nor lose: a multislice chain applies
a forward and an inverse transform per slice and direction, so a mean gain of a pair other than 1
(twiddle factors whose rounded magnitudes all fall on one side of 1) adds up over the slices, where
rounding errors of either sign average out. Over the elements the mean gain of a pair has to stay
within half a unit in the last place of 1, 2^-25 (the random part of the mean, 2e-7 / sqrt(65536)
per pair, is far below it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HALF_ULP = 2.0 ** -25


def _gain(x, y):
    x, y = x.cpu().numpy().astype(np.complex128), y.cpu().numpy().astype(np.complex128)
    return (np.vdot(x, y) / np.vdot(x, x)).real - 1


def _noise(shape):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(5)
    return torch.view_as_complex(torch.randn((*shape, 2), generator=gen, device="cuda"))


@pytest.mark.parametrize("W,n", [(64, 16), (128, 4), (256, 2)])
def test_window_pairs(W, n):
    from pypty_gb300.engine import Engine
    eng, x, pairs = Engine(), _noise((n, W, W)), 16
    y = x
    for _ in range(pairs):
        y = eng.fft2(eng.fft2(y), inverse=True)
    assert abs(_gain(x, y)) / pairs <= HALF_ULP


@pytest.mark.parametrize("ny,nx,K", [(64, 64, 16), (128, 256, 2), (512, 512, 1), (1024, 64, 1)])
def test_full_array_pairs(ny, nx, K):
    import torch
    from pypty_gb300.optim import fourier_clean_
    x, pairs = _noise((ny, nx, K)), 16
    ones = torch.ones((ny, nx), device="cuda")
    y = x.clone()
    for _ in range(pairs):
        fourier_clean_(y, mask=ones, out=y)
    assert abs(_gain(x, y)) / pairs <= HALF_ULP
