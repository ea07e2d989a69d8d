"""The one-patch-per-block step of the tiled forms: the bits of the
warp-per-tile step (taken when a tile shape is set), over direction counts
and ragged grids, resting and moving fluids, far departures and bands of
rows."""
import importlib

import numpy as np
import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")

FORMS = {"fp32": grlbm.PRECISION_FP32, "fast64": grlbm.FAST_FP64}
#        nx, ny, directions: remainders of the 8-cell runs, 32-pair passes and 4-direction stores
SIZES = [(8, 8, 32), (2, 2, 17), (9, 17, 20), (23, 7, 33), (41, 30, 50), (37, 26, 64), (16, 40, 96), (19, 21, 200), (130, 97, 36)]


def _case(nx, ny, nd, curved, moving):
    c = W.curved_scatter(nx_=nx, ny_=ny, n_dir=nd, n_fourier=5, steps=6)
    f = c["fields"]
    rng = np.random.default_rng(nx * 1000 + nd)
    n = f["eta"].size
    f["eta"] = rng.uniform(0.0, 1.0, n)
    if moving:
        f["ux"], f["uy"] = rng.uniform(-0.2, 0.2, n), rng.uniform(-0.2, 0.2, n)
        f["kappa1"] = rng.uniform(0.0, 0.3, n)
    if not curved:
        c.update(metric_kind=W.MINKOWSKI, streaming_type=W.FLAT_FIXED, excision=-1.0)
    return c


def _run(case, form, tile, I0):
    with grlbm.prepare(case, form) as r:
        if tile:
            r.set_tile_shape(*tile)
        r.set_intensity(I0)
        r.step(6)
        m = r.moments_if()
        return [r.intensity()] + [m[k] for k in sorted(m)] + [np.array(r.stats()["max_iterations"])]


@pytest.mark.gpu
@pytest.mark.parametrize("moving", [False, True])
@pytest.mark.parametrize("curved", [False, True])
@pytest.mark.parametrize("form", ["fp32", "fast64"])
@pytest.mark.parametrize("size", SIZES)
def test_same_bits_as_the_warp_per_tile_step(size, form, curved, moving):
    case = _case(*size, curved, moving)
    I0 = np.random.default_rng(7).uniform(0.0, 2.0, (case["fields"]["eta"].size, size[2]))
    for got, want in zip(_run(case, FORMS[form], None, I0), _run(case, FORMS[form], (2, 1), I0)):
        assert np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp32", "fast64"])
@pytest.mark.parametrize("curved", [False, True])
def test_far_departures(form, curved):
    case = _case(40, 24, 36, curved, False)
    case["cfl"] = 1.8
    I0 = np.random.default_rng(8).uniform(0.0, 2.0, (case["fields"]["eta"].size, 36))
    for got, want in zip(_run(case, FORMS[form], None, I0), _run(case, FORMS[form], (4, 2), I0)):
        assert np.array_equal(got, want)
