"""The adaptive FP32 step's staged-patch stream (larger grids) against its
row-by-row stream (bands of few rows): the same bits, at ragged tiles, odd
direction counts, departures beyond a cell and a grid with a hole."""
import importlib

import numpy as np
import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")


def _case(nx, ny, nd, nf, cfl):
    c = W.curved_scatter(nx_=nx, ny_=ny, n_dir=nd, n_fourier=nf, steps=1)
    c.update(streaming_type=W.CURVED_ADAPTIVE, cfl=cfl)
    rng = np.random.default_rng(nd)
    c["fields"]["eta"] = rng.uniform(0.0, 1.0, c["fields"]["eta"].size)
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nd,nf,cfl", [(161, 85, 33, 5, 0.9), (129, 100, 20, 16, 0.9), (97, 141, 7, 9, 0.9),
                                             (160, 96, 64, 5, 1.8)])
def test_patch_stream_gives_the_row_streams_bits(nx, ny, nd, nf, cfl):
    case = _case(nx, ny, nd, nf, cfl)
    I0 = np.random.default_rng(3).uniform(0.0, 2.0, (case["fields"]["eta"].size, nd))
    with grlbm.prepare(case, grlbm.PRECISION_FP32) as r:
        r.set_intensity(I0)
        r.step(1)
        whole = r.moments_if()
    # the same step in bands of rows small enough for the row-by-row stream
    nodes = np.arange((nx + 2) * (ny + 2)).reshape(ny + 2, nx + 2)
    for lo in range(1, ny + 1, 30):
        hi = min(lo + 30, ny + 1)
        with grlbm.prepare(case, grlbm.PRECISION_FP32) as r:
            r.set_intensity(I0)
            r.set_rows(lo, hi)
            r.step(1)
            band = r.moments_if()
        at = nodes[lo:hi, 1 : nx + 1]
        for k in whole:
            assert np.array_equal(whole[k][at], band[k][at]), (k, lo)
