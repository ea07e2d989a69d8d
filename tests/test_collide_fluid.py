"""Which kernel the plain form's collide runs for the fluid of the fields last
set: at more resident blocks where some of it moves or scatters
anisotropically, and without the column one direction earlier where it moves.
The bits against the oracle are test_plain_paths.py's and test_gpu_parity.py's."""
import importlib

import numpy as np
import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")


def _kernel(r):
    """(column, general) of the collide a step launches."""
    r.step(1)
    k = r.step_kernel()
    assert k["kernel"] == "plain"
    return bool(k["detail"] & 1), bool(k["detail"] & 2)


@pytest.mark.gpu
@pytest.mark.parametrize("nd", [32, 90, 91, 92])
@pytest.mark.parametrize("adaptive", [False, True])
def test_choice_by_fluid(nd, adaptive):
    case = W.curved_scatter(nx_=20, ny_=17, n_dir=nd, n_fourier=3, steps=1, rk_tol=1e-6)
    case.update(metric_kind=W.MINKOWSKI, streaming_type=W.FLAT_ADAPTIVE if adaptive else W.FLAT_FIXED, excision=-1.0)
    n = case["fields"]["eta"].size
    one = np.zeros(n)
    one[n // 2] = 0.1
    with grlbm.prepare(case, grlbm.PLAIN_FP64) as r:
        for name, general, most in ((None, False, 91), ("kappa1", True, 91), ("uy", True, 90), (None, False, 91)):
            f = dict(case["fields"])
            if name:
                f[name] = one
            r.set_fields(f)
            assert _kernel(r) == (nd <= most, general and nd <= most), (name, nd)
