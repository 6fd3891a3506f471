"""The band limit on both sides of each line of its rule for threads per block (lines of 256, 512 and 1024
points, together and apart), and the columns of masks that pass little: one entry in a column, in the
first and the last row, in columns of every 256, against NumPy in FP64 to 1e-6 (two complex64 transforms)."""
import numpy as np
import pytest

from golden_io import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx,K", [(512, 128, 11), (512, 128, 12), (512, 128, 19), (512, 64, 75), (1024, 64, 3), (1024, 128, 37),
                                     (64, 1024, 19), (64, 1024, 39), (256, 64, 57), (256, 64, 76), (64, 256, 80),
                                     (2048, 512, 1), (512, 2048, 1)])
def test_clean_threads(ny, nx, K):
    import torch
    from pypty_gb300.optim import fourier_clean_
    rng = np.random.default_rng(nx + K)
    x = (rng.normal(size=(ny, nx, K)) + 1j * rng.normal(size=(ny, nx, K))).astype(np.complex64)
    keep = np.zeros((ny, nx), np.float32)
    keep[rng.integers(0, ny, 60), rng.integers(0, nx, 60)] = rng.uniform(0.5, 1, 60)   # one entry in most columns
    keep[0, 3] = keep[ny - 1, 5] = keep[ny // 2, nx - 1] = keep[1, nx // 2] = 1.0
    f = np.fft.fft2(x.astype(np.complex128), axes=(0, 1))
    for mask in (keep, np.ones_like(keep)):
        got = fourier_clean_(torch.from_numpy(x).cuda(), mask=torch.from_numpy(np.fft.fftshift(mask)).cuda())
        assert rel_l2(got.cpu().numpy(), np.fft.ifft2(f * mask[:, :, None], axes=(0, 1))) <= 1e-6
