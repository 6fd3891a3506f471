"""The fused call run as forward half, loss and adjoint half (batches that fill the GPU) against
the whole-pass kernel (smaller batches) on the same positions: every position's gradient and
pattern bit for bit; loss, object and probe gradients, whose sums are grouped by batch, to the
rounding of those sums (2e-6 of the norm: a few hundred float32 terms per pixel)."""
import numpy as np
import pytest

from golden_io import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,n,batches,opts", [
    (64, 229, (229, 114), {}),                              # 458 and 228 blocks; just over what the GPU holds
    (64, 240, (240, 120), dict(edge_mult=1.5, smooth_rolloff=0.08)),
    (128, 58, (58, 57), {}),                                # 116 and 114 blocks: both sides of the line
    (128, 60, (60, 19), dict(step_pos=False, probe_shift=False, step_probe=False)),
    (128, 59, (59, 31), dict(step_obj=False, algorithm="ml")),
])
def test_halves_match_the_whole_pass(W, n, batches, opts):
    import torch
    from pypty_gb300 import synth
    from pypty_gb300.engine import Engine, Geometry, make_problem
    rng = np.random.default_rng(W + n)
    px, Z, Mp = 0.15, 3, 2
    pos = rng.uniform(0, 30, (n, 2))
    ipos, corr = synth.split_positions(pos)
    if opts.get("probe_shift", True) is False:
        corr[:] = 0
    ny, nx = W + 33, W + 41
    obj = np.exp(1j * rng.normal(0, 0.2, (ny, nx, Z, 1))).astype(np.complex64)
    probe = synth.make_probe(W, px, 300.0, 30.0, 60.0, Mp, [0.7, 0.3], 1e4)
    meas = rng.poisson(30.0, (n, W, W)).astype(np.float32)
    kw = dict(dict(algorithm="lsq_sqrt", step_pos=True), **opts)
    obj_d, probe_d, meas_d = (torch.from_numpy(a).cuda() for a in (obj, probe, meas))
    geo, out, sim = Geometry.make(ipos, corr), [], []
    for b in batches:
        prob = make_problem(W, obj.shape, Mp, geo, wavelength=synth.wavelength_A(300.0), pixel_size_x=px,
                            pixel_size_y=px, slice_distance=2.0, compute_batch=b, **kw)
        eng = Engine()
        out.append([t.cpu().numpy() for t in eng.loss_and_direction(prob, obj_d, probe_d, geo, meas_d)])
        sim.append(eng.simulate(prob, obj_d, probe_d, geo).cpu().numpy())
    (l0, o0, p0, g0), (l1, o1, p1, g1) = out
    assert np.isfinite(l0).all() and np.abs(l0 - l1).max() <= 1e-12 * np.abs(l1).max()
    assert np.array_equal(g0, g1) and np.array_equal(sim[0], sim[1])
    for a, b in ((o0, o1), (p0, p1)):
        assert (np.abs(b).max() == 0 and np.abs(a).max() == 0) or rel_l2(a, b) <= 2e-6
