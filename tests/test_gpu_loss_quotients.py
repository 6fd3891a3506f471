"""The loss's square roots and quotients without the library's slow paths (pixel values at the ends
of their range: zero, denormal, tiny, huge, infinite) against FP64, through one-slice patterns
whose intensity is set by the probe's scale. The amplitude loss and the quotient loss of a pixel
are within a few float32 roundings of the FP64 formula of the same intensities: 4e-6 relative
bounds a sum of W^2 of them, whose terms are float32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algorithm", ["lsq_sqrt", "lsq_sqrt_2"])
@pytest.mark.parametrize("modes", [1, 3])
@pytest.mark.parametrize("scale", [1e-22, 1e-12, 1.0, 1e12, 4e17])
def test_losses_over_the_range_of_intensities(algorithm, modes, scale):
    import torch
    from pypty_gb300 import synth
    from pypty_gb300.engine import Engine, Geometry, make_problem
    W, rng = 64, np.random.default_rng(2)
    probe = (synth.make_probe(W, 0.2, 200.0, 25.0, 60.0, modes, None, 1.0) * scale).astype(np.complex64)
    pos = np.array([[0, 0], [3, 5], [7, 1]])
    geo = Geometry.make(pos, np.zeros((3, 2), np.float32))
    obj = np.exp(1j * rng.normal(0, 0.3, (72, 72, 1, 1))).astype(np.complex64)
    prob = make_problem(W, obj.shape, modes, geo, algorithm=algorithm, wavelength=0.025, pixel_size_x=0.2,
                        pixel_size_y=0.2, slice_distance=1.0, step_pos=False, probe_shift=False)
    eng = Engine()
    obj_d, probe_d = torch.from_numpy(obj).cuda(), torch.from_numpy(probe).cuda()
    I = eng.simulate(prob, obj_d, probe_d, geo).cpu().numpy()
    M = (I * rng.uniform(0, 3, I.shape)).astype(np.float32)
    M[:, ::7] = 0
    ls, og, pg, _ = eng.loss_and_direction(prob, obj_d, probe_d, geo, torch.from_numpy(M).cuda())
    i, m = I.astype(np.float64), M.astype(np.float64)
    if algorithm == "lsq_sqrt":
        ref = ((np.sqrt(i) - np.sqrt(m)) ** 2).sum()
    else:
        big = m > 0.5
        ref = (0.5 * (i - m)[big] ** 2 / m[big]).sum() + i[~big].sum()
    got = float(ls[0])
    if (i - m).max() ** 2 > np.finfo(np.float32).max and algorithm == "lsq_sqrt_2":
        assert not np.isfinite(got)          # the squared error overflows float32, as it always did
    else:
        assert abs(got - ref) <= 4e-6 * abs(ref)
        assert np.isfinite(og.cpu().numpy()).all() and np.isfinite(pg.cpu().numpy()).all()
