"""The whole pass run as its halves keeps one pattern (dL/dI) per position of its buffers beside what the
same call would keep otherwise: a batch just over the line between the routes takes what its windows
take, not a far-field wave per mode more."""
import pytest

from pypty_gb300 import _lib, build


def _bytes(W, Z, Mp, batch, n=1200):
    p = _lib.Problem()
    for k, v in dict(window=W, obj_ny=1024, obj_nx=1024, n_slices=Z, n_obj_modes=1, n_probe_modes=Mp, n_positions=n,
                     n_sequence=n, compute_batch=batch, step_obj=1, step_probe=1, wavelength=0.02, pixel_size_x=0.1,
                     pixel_size_y=0.1, slice_distance=2.0, edge_mult=1.0, damping_cutoff=2 / 3, loss_weight=1.0).items():
        setattr(p, k, v)
    return _lib.workspace_bytes(p)


@pytest.mark.parametrize("W,line", [(64, 456), (128, 114)])
@pytest.mark.parametrize("Z,Mp", [(1, 2), (1, 4), (6, 3)])
def test_halves_workspace(W, line, Z, Mp):
    build.build()
    whole = line // Mp                           # blocks on the line: one pass
    slope = _bytes(W, Z, Mp, whole) - _bytes(W, Z, Mp, whole - 8)       # 8 positions more
    over = _bytes(W, Z, Mp, whole + 8) - _bytes(W, Z, Mp, whole)
    patterns = 2 * (whole + 8) * 4 * W * W       # dL/dI, two batches in flight
    assert over <= slope + patterns + 4096
    assert over >= slope + (whole + 8) * 4 * W * W     # the line is where this file says: dL/dI comes with it
