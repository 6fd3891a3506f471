"""128-px passes whose blocks walk runs of windows with the next one's load in flight: each window's
result is that of a call with the window alone, bit for bit, whatever its place in a run, and
transforms agree with NumPy's in FP64 to 1e-6 (a complex64 transform of 2^14 points: about 2e-7)."""
import numpy as np
import pytest

from golden_io import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,offset,inplace", [(1, 0, False), (152, 1, False), (153, 0, True), (457, 1, True)])
def test_fft_runs(n, offset, inplace):
    import torch
    from pypty_gb300.engine import Engine
    eng = Engine()
    g = torch.Generator(device="cuda").manual_seed(n)
    # offset: windows that do not start on 16 bytes
    store = torch.view_as_complex(torch.randn((n * 128 * 128 + offset, 2), device="cuda", generator=g))
    x = store[offset:].view(n, 128, 128)
    for inverse in (False, True):
        for shift in (False, True):
            want = torch.stack([eng.fft2(x[i:i + 1].clone(), inverse=inverse, shift=shift)[0] for i in range(n)])
            src = x.clone() if offset == 0 else store.clone()[offset:].view(n, 128, 128)
            got = eng.fft2(src, inverse=inverse, shift=shift, out=src if inplace else None)
            assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))
            for i in (0, n // 2, n - 1):
                a = x[i].cpu().numpy().astype(np.complex128)
                ref = (np.fft.ifft2(np.fft.ifftshift(a) if shift else a) if inverse
                       else np.fft.fftshift(np.fft.fft2(a)) if shift else np.fft.fft2(a))
                assert rel_l2(got[i].cpu().numpy(), ref) <= 1e-6


@pytest.mark.parametrize("Mp,nx", [(1, 170), (2, 169), (3, 171)])
def test_band_limit_runs(Mp, nx):
    """60 positions x 3 slices in one batch (runs of two windows, the last one short) against batches
    of 50 and of 1; loss and summed gradients to the rounding of their sums, grouped by batch."""
    import torch
    from pypty_gb300 import synth
    from pypty_gb300.engine import Engine, Geometry, make_problem
    rng = np.random.default_rng(nx)
    n, Z, px = 60, 3, 0.15
    ipos, corr = synth.split_positions(rng.uniform(0, 30, (n, 2)))
    obj = np.exp(1j * rng.normal(0, 0.2, (163, nx, Z, 1))).astype(np.complex64)
    probe = synth.make_probe(128, px, 300.0, 30.0, 60.0, Mp, np.arange(Mp, 0, -1), 1e4)
    meas = torch.from_numpy(rng.poisson(30.0, (n, 128, 128)).astype(np.float32)).cuda()
    obj_d, probe_d = torch.from_numpy(obj).cuda(), torch.from_numpy(probe).cuda()
    geo, eng, out = Geometry.make(ipos, corr), Engine(), []
    for b in (60, 50, 1):
        prob = make_problem(128, obj.shape, Mp, geo, algorithm="lsq_sqrt", wavelength=synth.wavelength_A(300.0),
                            pixel_size_x=px, pixel_size_y=px, slice_distance=2.0, compute_batch=b, step_pos=True)
        r = [t.cpu().numpy() for t in eng.loss_and_direction(prob, obj_d, probe_d, geo, meas)]
        out.append(r + [eng.simulate(prob, obj_d, probe_d, geo).cpu().numpy()])
    l0, o0, p0, g0, s0 = out[0]
    for l1, o1, p1, g1, s1 in out[1:]:
        assert np.array_equal(s0, s1) and np.array_equal(g0, g1)
        assert np.abs(l0 - l1).max() <= 1e-12 * np.abs(l1).max()
        assert rel_l2(o0, o1) <= 2e-6 and rel_l2(p0, p1) <= 2e-6


@pytest.mark.parametrize("axes,order", [((1, 2), (0, 1, 2)), ((-2, -1), (2, 1, 0)), ((0, 1), (1, 2, 0)), ((2, 1), (0, 2, 1)),
                                        ((2, 0), (2, 0, 1))])
def test_fft_wrapper_axes(axes, order):
    """The wrapper's axes, last two or not, of contiguous and permuted tensors against NumPy."""
    import torch
    from pypty_gb300 import fft
    rng = np.random.default_rng(3)
    shape = [64, 64, 64]
    other = ({0, 1, 2} - {a % 3 for a in axes}).pop()
    shape[other] = 3
    mem = [shape[i] for i in order]                     # the tensor's axis order in memory
    a = (rng.normal(size=mem) + 1j * rng.normal(size=mem)).astype(np.complex64).transpose(np.argsort(order))
    t = torch.from_numpy(np.ascontiguousarray(a.transpose(order))).cuda().permute(*np.argsort(order).tolist())
    assert tuple(t.shape) == tuple(shape)
    for f, g in ((fft.fft2, np.fft.fft2), (fft.ifft2, np.fft.ifft2)):
        got = f(t, axes=axes)
        assert got.is_contiguous()
        assert rel_l2(got.cpu().numpy(), g(a.astype(np.complex128), axes=axes)) <= 1e-6
