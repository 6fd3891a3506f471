"""Band limit of full arrays by lines of 64 to 1024 points: both block sizes, lines that do not fill
a block, odd and even line strides, masks with empty and single columns, in place, with a step,
against NumPy in FP64 to 1e-6 (two complex64 transforms of up to 2^20 points: about 3e-7); a NaN
spreads over its slice and no further."""
import numpy as np
import pytest

from golden_io import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx,K,kind", [(64, 64, 3, "band"), (128, 256, 1, "given"), (256, 128, 77, "band"),
                                          (512, 64, 21, "given"), (64, 512, 5, "roll"), (1024, 64, 2, "given"),
                                          (256, 1024, 13, "band"), (512, 512, 20, "given"), (64, 2048, 1, "band"),
                                          (2048, 64, 3, "given")])
def test_clean_lines(ny, nx, K, kind):
    import torch
    from pypty_gb300.optim import fourier_clean_
    rng = np.random.default_rng(ny + nx + K)
    x, dx = (rng.normal(size=(ny, nx, K)) + 1j * rng.normal(size=(ny, nx, K)) for _ in range(2))
    x, dx = x.astype(np.complex64), dx.astype(np.complex64)
    fy, fx = np.meshgrid(np.fft.fftfreq(ny), np.fft.fftfreq(nx), indexing="ij")
    r = fx ** 2 + fy ** 2
    kw = dict(cutoff=0.6)
    mask = (r <= np.float32(np.float32(0.3) * np.float32(0.3))).astype(np.float64)
    if kind == "roll":
        kw["rolloff"] = 0.2
        r0, r1 = float(np.float32(0.2) ** 2), float(np.float32(0.3) ** 2)
        t = 0.5 * (1 + np.cos(np.pi * (r - r0) / (r1 - r0)))
        mask = np.where(r > r0, mask * t, mask)
    elif kind == "given":
        m = rng.uniform(0, 1, (ny, nx)).astype(np.float32)
        m[:, ::3] = 0
        m[:, 1] = 0
        m[3, 1] = 0.5               # one entry of a column
        m[:, nx // 2:nx // 2 + 7] = 0   # in shifted order: kx = 0 and its neighbours
        kw, mask = dict(mask=torch.from_numpy(m).cuda()), np.fft.ifftshift(m).astype(np.float64)
    def ref(a):
        return np.fft.ifft2(np.fft.fft2(a.astype(np.complex128), axes=(0, 1)) * mask[:, :, None], axes=(0, 1))
    xd, dxd = torch.from_numpy(x).cuda(), torch.from_numpy(dx).cuda()
    out = torch.full_like(xd, float("nan"))
    fourier_clean_(xd, out=out, **kw)
    assert rel_l2(out.cpu().numpy(), ref(x)) <= 1e-6
    fourier_clean_(xd, out=out, dx=dxd, step=0.3, **kw)
    assert rel_l2(out.cpu().numpy(), ref(x + np.float32(0.3) * dx)) <= 1e-6
    y = xd.clone()
    fourier_clean_(y, out=y, **kw)
    assert rel_l2(y.cpu().numpy(), ref(x)) <= 1e-6
    y = xd.clone()
    y[ny // 2, 1, K - 1] = float("nan")
    fourier_clean_(y, out=out, **kw)
    bad = torch.isnan(torch.view_as_real(out)).any(-1)
    assert bad[:, :, K - 1].all() and not bad[:, :, :K - 1].any()
