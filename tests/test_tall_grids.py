"""Grids of more rows than one launch's grid holds along y: 65535 rows of 8
cells of the block step, and of 2 cells of the adaptive patch stream."""
import importlib

import numpy as np
import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["PRECISION_FP32", "FAST_FP64"])
def test_block_step(form):
    ny = 65535 * 8 + 13
    case = W.flat_beam(nx_=2, ny_=ny, n_dir=4, steps=2)
    case["keep_source_nodes_active"] = 0
    I0 = W.uniform(3, (ny + 2) * 4 * 4)

    def run(tile):
        with grlbm.Radiation(case, getattr(grlbm, form)) as r:
            if tile:
                r.set_tile_shape(*tile)
            r.set_intensity(I0)
            r.step(2)
            return [r.intensity()] + list(r.moments_if().values())

    for a, b in zip(run(None), run((2, 8))):
        assert np.array_equal(a, b)
    assert np.any(a[-40:] != 0)


@pytest.mark.gpu
def test_adaptive_patch_stream():
    """Against the row-by-row stream, which a band of few rows takes."""
    ny, nd = 65535 * 2 + 11, 8
    case = W.curved_scatter(nx_=2, ny_=ny, n_dir=nd, n_fourier=3, steps=1, rk_tol=1e-6)
    case.update(streaming_type=W.CURVED_ADAPTIVE)
    I0 = W.uniform(4, (ny + 2) * 4 * nd)
    with grlbm.prepare(case, grlbm.PRECISION_FP32) as r:
        r.set_intensity(I0)
        r.step(1)
        whole = r.moments_if()
    lo = ny - 60
    with grlbm.prepare(case, grlbm.PRECISION_FP32, rows=(lo, ny + 1)) as r:
        r.set_intensity(I0)
        r.step(1)
        band = r.moments_if()
    for k in whole:
        a, b = (m[k].reshape(ny + 2, 4)[lo : ny + 1, 1:3] for m in (whole, band))
        assert np.array_equal(a, b), k
        assert k != "E" or np.all(a > 0)
