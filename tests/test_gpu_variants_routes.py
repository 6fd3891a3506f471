"""The variants path on both sides of the line in slices from which on it runs on the fused kernel's halves
(by window, object modes, probe modes, batch and tilt gradient), against the FP64 oracle. Bounds: the
complex64 tolerances (loss 1e-5, gradients 1e-4), or 1.5 times the error of the oracle's own complex64
arithmetic where that is larger."""
import numpy as np
import pytest

from test_gpu_variants import errors, fp64_variant_oracle, run_gpu_variant
from test_gpu_variants_fused import make_case

pytestmark = pytest.mark.gpu

NEAR = dict(recon_type="near_field", defocus=80.0)


@pytest.mark.parametrize("c", [
    dict(W=64, Z=1, Mp=2, Mo=1, n=7, batch=4, **NEAR), dict(W=64, Z=1, Mp=2, Mo=1, n=125, batch=122, **NEAR),
    dict(W=64, Z=2, Mp=3, Mo=1, n=5, batch=5, tilt_mode=3, rows=True), dict(W=64, Z=2, Mp=1, Mo=2, n=5, batch=3, tilt_mode=0, rows=True),
    dict(W=64, Z=3, Mp=1, Mo=2, n=5, batch=3, **NEAR), dict(W=128, Z=1, Mp=1, Mo=1, n=4, batch=4, tilt_mode=4, rows=True),
    dict(W=128, Z=3, Mp=2, Mo=2, n=3, batch=2, **NEAR), dict(W=128, Z=3, Mp=2, Mo=2, n=3, batch=2, tilt_mode=4, rows=True),
    dict(W=128, Z=4, Mp=1, Mo=3, n=3, batch=3, **NEAR), dict(W=128, Z=4, Mp=3, Mo=2, n=2, batch=2, tilt_mode=0, rows=True),
    dict(W=128, Z=5, Mp=4, Mo=2, n=2, batch=2, **NEAR), dict(W=128, Z=6, Mp=4, Mo=2, n=2, batch=2, **NEAR),
], ids=lambda c: "-".join("%s%s" % kv for kv in c.items() if kv[0] in ("W", "Z", "Mp", "Mo", "n", "tilt_mode")))
def test_both_sides_of_the_line(c):
    c = make_case(**c)
    o64, o32 = fp64_variant_oracle(c), fp64_variant_oracle(c, np.float32, np.complex64)
    kept = (lambda r: list(r)) if c["step_tilts"] else (lambda r: list(r)[:7] + [None] + list(r)[8:])
    e, floor = errors(kept(run_gpu_variant(c)), kept(o64)), errors(kept(o32), kept(o64))
    assert {"loss", "pos"} <= set(e)
    for k, v in e.items():
        assert v <= max(1e-5 if k == "loss" else 1e-4, 1.5 * floor.get(k, 0.0)), (k, v, floor.get(k))
