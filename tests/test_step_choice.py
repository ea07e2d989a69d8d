"""Which kernel the default step of the tiled forms runs: one patch per block
up to a number of cells that depends on the form and the directions, warps with
a tile each from there on, both for the rows of each launch -- and the same
bits on either side, whole or in bands of rows."""
import importlib

import numpy as np
import pytest
import torch

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")

pytestmark = pytest.mark.gpu
FORMS = {"fp32": grlbm.PRECISION_FP32, "fast64": grlbm.FAST_FP64}


def _case(nx, ny, nd, curved, moving=False, cfl=0.9):
    c = W.curved_scatter(nx_=nx, ny_=ny, n_dir=nd, n_fourier=5, steps=2, rk_tol=1e-8)
    f = c["fields"]
    rng = np.random.default_rng(nx * 1000 + nd)
    n = f["eta"].size
    f["eta"] = rng.uniform(0.0, 1.0, n)
    if moving:
        f["ux"], f["uy"] = rng.uniform(-0.2, 0.2, n), rng.uniform(-0.2, 0.2, n)
        f["kappa1"] = rng.uniform(0.0, 0.3, n)
    if not curved:
        c.update(metric_kind=W.MINKOWSKI, streaming_type=W.FLAT_FIXED, excision=-1.0)
    c["cfl"] = cfl
    return c


def _kernel(r, step):
    """What the step that `step` enqueues last runs: 8 or 4, the cells of a run
    of the one-patch-per-block kernel, or "warp"."""
    step()
    k = r.step_kernel()
    return k["detail"] if k["kernel"] == "block" else k["kernel"]


def _result(r, I0, steps=2):
    r.set_intensity(I0)
    r.step(steps)
    m = r.moments_if()
    return [r.intensity()] + [m[k] for k in sorted(m)]


# on both sides of each line of the rule
@pytest.mark.parametrize("form,curved,nd,nx,ny,warp", [
    ("fp32", False, 4, 250, 238, False), ("fp32", False, 4, 250, 242, True),
    ("fp32", False, 8, 330, 330, False), ("fp32", False, 8, 340, 330, True),
    ("fp32", False, 33, 300, 299, False), ("fp32", False, 33, 301, 301, True),
    ("fp32", False, 32, 400, 399, False), ("fp32", False, 32, 401, 400, True),
    ("fp32", False, 64, 400, 400, False), ("fp32", False, 72, 560, 560, False),
    ("fp32", True, 12, 316, 316, False), ("fp32", True, 12, 317, 317, True),
    ("fp32", True, 20, 400, 400, False), ("fp32", True, 28, 346, 346, False), ("fp32", True, 28, 347, 347, True),
    ("fast64", True, 32, 316, 316, False), ("fast64", True, 32, 317, 317, True),
    ("fast64", True, 24, 400, 400, False), ("fast64", True, 33, 400, 400, False), ("fast64", False, 32, 600, 600, False)])
def test_choice_and_bits(form, curved, nd, nx, ny, warp):
    case = _case(nx, ny, nd, curved)
    with grlbm.prepare(case, FORMS[form]) as r:
        assert _kernel(r, lambda: r.step(1)) == ("warp" if warp else 8)
        # a third of the rows at a time: the block step
        third = 1 + ny // 3
        assert _kernel(r, lambda: r.step_rows_async(1, 1 + third, True)) == 8
        # an edge row: runs of 4 up to one 8-cell tile for every second SM
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        assert _kernel(r, lambda: r.step_rows_async(1, 2, True)) == (4 if 2 * -(-nx // 8) <= sms else 8)
        r.sync()
        I0 = np.random.default_rng(nd).uniform(0.0, 2.0, case["fields"]["eta"].size * nd)
        whole = _result(r, I0, 1)
        r.set_intensity(I0)
        for lo in range(1, ny + 1, third):
            r.step_rows_async(lo, min(lo + third, ny + 1), lo + third > ny)
        r.sync()
        parts = [r.intensity()] + [m for _, m in sorted(r.moments_if().items())]
        for a, b in zip(whole, parts):
            assert np.array_equal(a, b)


# runs of 8: remainders of runs, 32-pair passes and rows of tiles, each width
# of store, and departures of more than a cell
@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("form", ["fp32", "fast64"])
@pytest.mark.parametrize("nx,ny,nd", [(101, 67, 17), (77, 83, 33), (91, 70, 50), (99, 75, 64)])
def test_runs_of_eight(form, nx, ny, nd, curved, moving):
    case = _case(nx, ny, nd, curved, moving)
    I0 = np.random.default_rng(7).uniform(0.0, 2.0, case["fields"]["eta"].size * nd)
    with grlbm.prepare(case, FORMS[form]) as r:
        assert _kernel(r, lambda: r.step(1)) == 8
        got = _result(r, I0, 4)
        r.set_tile_shape(2, 1)
        assert _kernel(r, lambda: r.step(1)) == "warp"
        want = _result(r, I0, 4)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("form", ["fp32", "fast64"])
def test_far_departures_in_runs_of_eight(form, curved):
    case = _case(90, 81, 36, curved, cfl=1.8)
    I0 = np.random.default_rng(8).uniform(0.0, 2.0, case["fields"]["eta"].size * 36)
    with grlbm.prepare(case, FORMS[form]) as r:
        assert _kernel(r, lambda: r.step(1)) == 8
        got = _result(r, I0, 4)
        r.set_tile_shape(4, 2)
        want = _result(r, I0, 4)
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("form", ["fp32", "fast64"])
def test_bands_of_rows(form, curved):
    nx, ny, nd = 85, 93, 24
    case = _case(nx, ny, nd, curved)
    I0 = np.random.default_rng(9).uniform(0.0, 2.0, case["fields"]["eta"].size * nd)
    with grlbm.prepare(case, FORMS[form]) as r:
        whole = _result(r, I0, 1)
    nodes = np.arange((nx + 2) * (ny + 2)).reshape(ny + 2, nx + 2)
    for lo, hi in ((1, 12), (12, 75), (75, 76), (76, ny + 1)):
        with grlbm.prepare(case, FORMS[form], rows=(lo, hi)) as r:
            band = _result(r, I0, 1)
        at = nodes[lo:hi, 1 : nx + 1]
        assert np.array_equal(whole[0].reshape(-1, nd)[at], band[0].reshape(-1, nd)[at])
        for a, b in zip(whole[1:], band[1:]):
            assert np.array_equal(a[at], b[at])
