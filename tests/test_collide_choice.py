"""Which kernel the plain form's collide runs: the cells' streamed values in a
column of shared memory up to 91 directions.  The bits against the oracle are test_plain_paths.py's."""
import importlib

import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")


def _column(r):
    """Whether the collide that a step launches has the column."""
    r.step(1)
    k = r.step_kernel()
    assert k["kernel"] == "plain"
    return bool(k["detail"] & 1)


@pytest.mark.gpu
@pytest.mark.parametrize("nd", [32, 90, 91, 92])
@pytest.mark.parametrize("adaptive", [False, True])
def test_column_by_directions(nd, adaptive):
    case = W.curved_scatter(nx_=20, ny_=17, n_dir=nd, n_fourier=3, steps=1, rk_tol=1e-6)
    case.update(metric_kind=W.MINKOWSKI, streaming_type=W.FLAT_ADAPTIVE if adaptive else W.FLAT_FIXED, excision=-1.0)
    with grlbm.prepare(case, grlbm.PLAIN_FP64) as r:
        assert _column(r) == (nd <= 91)
