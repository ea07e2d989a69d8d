"""The tile in force, what it is reported as, and the way back to the default
step, also after a batch has been autotuned."""
import importlib

import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")

pytestmark = pytest.mark.gpu
FORMS = {"fp32": grlbm.PRECISION_FP32, "fast64": grlbm.FAST_FP64}


def _case(n, nd):
    return W.curved_scatter(nx_=n, ny_=n, n_dir=nd, n_fourier=5, steps=1)


def _runs_block_step(r):
    r.step(1)
    return r.step_kernel()["kernel"] == "block"


@pytest.mark.parametrize("form", ["fp32", "fast64"])
def test_reported_tile_is_the_one_in_force(form):
    with grlbm.prepare(_case(40, 24), FORMS[form]) as r:
        assert r.tile_shape() == (0, 0) and _runs_block_step(r)
        r.set_tile_shape(4, 2)
        assert r.tile_shape() == (4, 2) and not _runs_block_step(r)
        for bad in ((0, 3), (3, 0), (-1, 1), (17, 1)):
            with pytest.raises(grlbm.GrlbmError):
                r.set_tile_shape(*bad)
            assert r.tile_shape() == (4, 2)
        r.set_tile_shape(0, 0)
        assert r.tile_shape() == (0, 0) and _runs_block_step(r)
        r.set_tile_shape(*r.tile_shape())
        assert _runs_block_step(r)


@pytest.mark.parametrize("form", ["fp32", "fast64"])
def test_autotuned_problems_report_what_they_run(form):
    probs = [grlbm.prepare(_case(n, nd), FORMS[form]) for n, nd in ((64, 16), (96, 24), (48, 32))]
    try:
        with grlbm.Batch(probs) as b:
            choice = b.autotune(2)
        for r in probs:
            block = _runs_block_step(r)
            assert block if choice["blocks_per_sm"] > 0 else block == (r.tile_shape() == (0, 0))
    finally:
        for r in probs:
            r.close()
