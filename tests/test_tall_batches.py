"""Grids of more rows of tiles than one launch's grid holds along y, in a
batch: the block step in several launches, and on a share, against the
warp-per-tile step that such a grid takes alone."""
import importlib

import numpy as np
import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [0, -1])
def test_block_step(shape):
    ny = 65535 * 8 + 13
    case = W.flat_beam(nx_=2, ny_=ny, n_dir=4, steps=2)
    case["keep_source_nodes_active"] = 0
    I0 = W.uniform(3, (ny + 2) * 4 * 4)
    with grlbm.Radiation(case, grlbm.PRECISION_FP32) as r:
        r.set_intensity(I0)
        r.step(2)
        assert r.step_kernel()["kernel"] == "warp"
        want = [r.intensity()] + list(r.moments_if().values())
        r.set_intensity(I0)
        with grlbm.Batch([r]) as b:
            b.set_shape(shape)
            b.step(2)
        k = r.step_kernel()
        assert k["kernel"] == "block" and (k["blocks"] == 65537 if shape == 0 else k["blocks"] < 65537)
        got = [r.intensity()] + list(r.moments_if().values())
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    assert np.any(got[0][-40:] != 0)
