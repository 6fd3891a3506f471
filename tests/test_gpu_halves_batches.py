"""Several batches run as halves, two of them in flight on their own buffers and the last one short,
against the whole-pass kernel in smaller batches: every position's gradient and pattern bit for bit; loss,
object and probe gradients to the rounding of sums grouped by batch (2e-6 of the norm). Which side of the
line a batch is on is asked of the plan: only the halves keep a pattern per position (4 W^2 bytes) more."""
import numpy as np
import pytest

from golden_io import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,Z,n,batch,small,opts", [
    (64, 2, 499, 229, 114, {}),                                  # 458 blocks twice, then 82
    (64, 3, 470, 230, 100, dict(smooth_rolloff=0.08, algorithm="lsq_sqrt_2")),
    (128, 3, 121, 58, 40, {}),                                   # 116 blocks twice, then 10
    (128, 1, 179, 60, 57, dict(algorithm="ml", edge_mult=1.5)),
])
def test_several_batches_as_halves(W, Z, n, batch, small, opts):
    import torch
    from pypty_gb300 import _lib, synth
    from pypty_gb300.engine import Engine, Geometry, make_problem
    rng = np.random.default_rng(n)
    Mp = 2
    ipos, corr = synth.split_positions(rng.uniform(0, 30, (n, 2)))
    obj = np.exp(1j * rng.normal(0, 0.2, (W + 33, W + 41, Z, 1))).astype(np.complex64)
    probe = synth.make_probe(W, 0.15, 300.0, 30.0, 60.0, Mp, [0.7, 0.3], 1e4)
    meas = rng.poisson(30.0, (n, W, W)).astype(np.float32)
    kw = dict(dict(algorithm="lsq_sqrt", step_pos=True), **opts)
    obj_d, probe_d, meas_d = (torch.from_numpy(a).cuda() for a in (obj, probe, meas))
    geo, eng = Geometry.make(ipos, corr), Engine()

    def problem(b):
        return make_problem(W, obj.shape, Mp, geo, wavelength=synth.wavelength_A(300.0), pixel_size_x=0.15,
                            pixel_size_y=0.15, slice_distance=2.0, compute_batch=b, **kw)

    def extra(b):   # bytes of four more positions beyond their windows (object, waves, gradients, probes)
        windows = 4 * 2 * 8 * W * W * (Z + 2 * Z * Mp + Mp)
        return _lib.workspace_bytes(problem(b)) - _lib.workspace_bytes(problem(b - 4)) - windows

    line = (456 if W == 64 else 114) // Mp
    assert small <= line < batch and extra(line + 4) > line * 4 * W * W > extra(line)
    out, sim = [], []
    for b in (batch, small):
        out.append([t.cpu().numpy() for t in eng.loss_and_direction(problem(b), obj_d, probe_d, geo, meas_d)])
        sim.append(eng.simulate(problem(b), obj_d, probe_d, geo).cpu().numpy())
    (l0, o0, p0, g0), (l1, o1, p1, g1) = out
    assert np.isfinite(l0).all() and np.abs(l0 - l1).max() <= 1e-12 * np.abs(l1).max()
    assert np.array_equal(g0, g1) and np.array_equal(sim[0], sim[1])
    assert rel_l2(o0, o1) <= 2e-6 and rel_l2(p0, p1) <= 2e-6
