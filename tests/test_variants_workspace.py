"""The variants path keeps what the layered path keeps, and no window more per probe mode: its gradient
contributions take the places of the wave stack. On top come a pattern per position, the tables of the
variant and the partial tiles of a grouped scatter (two blocks for each of 152 SMs, 8 KB a tile)."""
import ctypes

import pytest

from pypty_gb300 import _lib, build


@pytest.mark.parametrize("W", [64, 128])
@pytest.mark.parametrize("Mp,Mo", [(1, 1), (3, 1), (8, 1), (4, 2), (1, 4)])
@pytest.mark.parametrize("Z,batch", [(1, 16), (6, 64), (20, 96)])
def test_variants_workspace(W, Mp, Mo, Z, batch):
    build.build()
    p = _lib.Problem()
    for k, v in dict(window=W, obj_ny=400, obj_nx=300, n_slices=Z, n_obj_modes=Mo, n_probe_modes=Mp, n_positions=200,
                     n_sequence=200, compute_batch=batch, step_obj=1, step_probe=1, wavelength=0.02, pixel_size_x=0.1,
                     pixel_size_y=0.1, slice_distance=2.0, edge_mult=1.0, damping_cutoff=2 / 3, loss_weight=1.0).items():
        setattr(p, k, v)
    v = _lib.Variant(recon_type=_lib.RECON_TYPES["near_field"], defocus=50.0, data_multiplier=1.0, upsample_pattern=1)
    layered, variants = ctypes.c_size_t(0), ctypes.c_size_t(0)
    lib = _lib.lib()
    assert lib.pty_layered_workspace_bytes(ctypes.byref(p), _lib.DFT_ENGINES["fp32_fft"], ctypes.byref(layered)) == 0
    assert lib.pty_variants_workspace_bytes(ctypes.byref(p), ctypes.byref(v), ctypes.byref(variants)) == 0
    patterns, tables, partial = 4 * batch * W * W, 1 << 20, (304 + 13 * 10 * Z * Mo) * 8192
    assert variants.value <= layered.value + patterns + tables + partial
