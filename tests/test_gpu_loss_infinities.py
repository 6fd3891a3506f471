"""Infinite operands of the quotient loss, on every route that forms it (whole pass, halves, 256-px
kernels, variants). dL/dI = I / M - 1 is -1 both for a measured value of 1e30 and for an infinite one, so
both give the same gradients bit for bit; a squared error that overflows float32 makes the loss +inf where
the sums are 64-bit numbers (256 px, variants), and not finite where they are compensated pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("route,W,n,modes", [("whole", 64, 3, 1), ("whole", 64, 3, 2), ("halves", 64, 230, 2),
                                             ("whole", 128, 2, 2), ("halves", 128, 58, 2), ("cluster", 256, 2, 2),
                                             ("near", 64, 3, 2), ("near", 256, 1, 1)])
def test_infinite_measurements(route, W, n, modes):
    import torch
    from pypty_gb300 import synth
    from pypty_gb300.engine import Engine, Geometry, make_problem
    rng = np.random.default_rng(W + n)
    pos = rng.integers(0, 8, (n, 2))
    geo = Geometry.make(pos, np.zeros((n, 2), np.float32))
    obj = np.exp(1j * rng.normal(0, 0.3, (W + 8, W + 8, 1, 1))).astype(np.complex64)
    probe = synth.make_probe(W, 0.2, 200.0, 25.0, 60.0, modes, None, 1e4).astype(np.complex64)
    prob = make_problem(W, obj.shape, modes, geo, algorithm="lsq_sqrt_2", wavelength=0.025, pixel_size_x=0.2,
                        pixel_size_y=0.2, slice_distance=1.0, step_pos=False, probe_shift=False, compute_batch=n)
    eng = Engine()
    obj_d, probe_d = torch.from_numpy(obj).cuda(), torch.from_numpy(probe).cuda()
    M = rng.poisson(3.0, (n, W, W)).astype(np.float32)

    def call(value):
        m = M.copy()
        m[0, W // 2 + 1, W // 2 - 2] = value
        m = torch.from_numpy(m).cuda()
        if route == "near":
            r = eng.loss_and_direction_variants(prob, obj_d, probe_d, geo, m, recon_type="near_field", defocus=50.0)
        else:
            r = eng.loss_and_direction(prob, obj_d, probe_d, geo, m)
        return [t.cpu().numpy() for t in r[:3]]

    _, o_big, p_big = call(1e30)
    _, o_inf, p_inf = call(np.inf)
    assert np.isfinite(o_big).all() and np.abs(p_big).max() > 0
    assert np.array_equal(o_inf, o_big) and np.array_equal(p_inf, p_big)
    loss, _, _ = call(1e25)
    if W == 256 or route == "near":
        assert np.isposinf(loss).all()
    else:
        assert not np.isfinite(loss).any()
