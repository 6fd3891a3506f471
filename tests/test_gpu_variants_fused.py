"""The variants path on the fused kernel's halves, at the edges of its routes, against the FP64
oracle: incoherent object modes with an edge propagator per position and a rolled-off mask in
ragged batches; more sequence entries than one pass of the tilt rows' sums, with a grouped
scatter; step propagators with a single tilt; more steps than one launch's weights; eight probe modes at one slice; no object gradient.

Bounds: the complex64 tolerances (loss 1e-5, gradients 1e-4), or 1.5 times the error of the
oracle's own complex64 arithmetic where that is larger."""
import numpy as np
import pytest

from test_gpu_variants import errors, fp64_variant_oracle, run_gpu_variant

pytestmark = pytest.mark.gpu

CASES = {
    "modes_edge_rolloff": dict(W=64, Z=3, Mp=2, Mo=2, n=13, batch=5, tilt_mode=4, rows=True, edge_mult=1.5, rolloff=0.08),
    "many_rows": dict(W=64, Z=2, Mp=1, Mo=1, n=300, batch=128, tilt_mode=3, rows=True),
    "steps_single_tilt": dict(W=128, Z=4, Mp=3, Mo=1, n=3, batch=1, tilt_mode=0, distances=[2.0, 1.5, 2.5, 3.0]),
    "many_steps": dict(W=64, Z=67, Mp=1, Mo=1, n=3, batch=2, tilt_mode=0, rows=True),
    "near_eight_modes": dict(W=64, Z=1, Mp=8, Mo=1, n=3, batch=2, recon_type="near_field", defocus=80.0, step_probe=0),
    "near_no_object": dict(W=128, Z=3, Mp=2, Mo=1, n=5, batch=5, recon_type="near_field", defocus=80.0, step_obj=0),
}


def make_case(W, Z, Mp, Mo, n, batch, tilt_mode=None, rows=False, **kw):
    from oracle import variants_oracle as vor
    from pypty_gb300 import synth
    rng = np.random.default_rng(W + n)
    px = 0.15
    ipos, corr = synth.split_positions(rng.uniform(0, 40, (n, 2)))
    c = dict(dict(distance=2.0, distances=None, edge_mult=1.0, wavelength=synth.wavelength_A(300.0), px=px, cutoff=2 / 3,
                  rolloff=0.0, loss_weight=1.0, batch=batch, step_probe=1, step_obj=1, step_pos=1, defocus=0.0, cs=0.0,
                  tan_x=0.0, tan_y=0.0, step_bc=0, step_ab=0, data_pad=0, use_padded=1, shift0=0, shift1=0, mult=1.0,
                  upsample=1, step_sb=0, algorithm="lsq_sqrt", recon_type="far_field", positions=ipos,
                  pos_correction=corr, sequence=np.arange(n)), **kw)
    for k in ("masks", "beam_current", "aberrations", "aberration_marker", "static_background", "defocus_array",
              "probe_marker"):
        c[k] = None
    c["tilt_mode"] = tilt_mode or 0
    c["tilts"] = None if tilt_mode is None else rng.normal(0, 5e-4, (n if rows else 1, 6)).astype(np.float32)
    c["step_tilts"] = int(tilt_mode is not None)
    c["obj"] = np.exp(1j * rng.normal(0, 0.2 / np.sqrt(Z), (W + 41, W + 45, Z, Mo))).astype(np.complex64)
    c["probe"] = synth.make_probe(W, px, 300.0, 30.0, 60.0, Mp, np.arange(Mp, 0, -1), 1e4)
    I = vor.loss_and_direction_variants(
        c["obj"], c["probe"], ipos, corr, c["distance"] if c["distances"] is None else c["distances"], c["edge_mult"],
        np.zeros((n, W, W), np.float32), c["algorithm"], c["wavelength"], 0, 0, 0, px, px, c["cutoff"], c["rolloff"],
        c["sequence"], 1.0, batch, recon_type=c["recon_type"], defocus=c["defocus"], tilts=c["tilts"],
        tilt_mode=c["tilt_mode"], simulate=True)
    c["measured"] = (np.asarray(I) * rng.uniform(0.6, 1.4, I.shape)).astype(np.float32)
    return c


@pytest.mark.parametrize("name", sorted(CASES))
def test_variants_fused_against_fp64_oracle(name):
    c = make_case(**CASES[name])
    o64, o32 = fp64_variant_oracle(c), fp64_variant_oracle(c, np.float32, np.complex64)
    def kept(r):
        r = list(r)
        for k, on in ((2, c["step_obj"]), (3, c["step_probe"]), (7, c["step_tilts"])):
            if not on:
                r[k] = np.ones(np.shape(r[k])) if k < 7 else None
        return r
    e = errors(kept(run_gpu_variant(c)), kept(o64))
    floor = errors(kept(o32), kept(o64))
    print(name, {k: "%.1e (complex64 %.1e)" % (v, floor.get(k, 0.0)) for k, v in e.items()})
    assert {"loss", "pos"} <= set(e)
    for k, v in e.items():
        assert v <= max(1e-5 if k == "loss" else 1e-4, 1.5 * floor.get(k, 0.0)), (k, v, floor.get(k))
