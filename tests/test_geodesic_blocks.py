"""The geodesic kernel's blocks (a run of cells of one row, up to 128 threads)
at their edges: direction counts that fill a block, leave threads idle or limit
its cells, rows shorter than a run, and backtraces that leave the staged node
rows -- coefficients against the oracle's at the table contract's bound."""
import numpy as np
import pytest
from conftest import rel_l2

COEF = ("coefS", "coefX", "coefY", "coefCx", "coefCy")


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nf,cfl", [(2, 3, 5, 0.9), (33, 20, 3, 0.9), (25, 26, 5, 0.9), (40, 17, 16, 0.9),
                                          (19, 18, 33, 0.9), (15, 22, 64, 0.9), (24, 24, 9, 2.3)])
def test_coefficients_match_the_oracle(grlbm, W, oracle, nx, ny, nf, cfl):
    c = W.curved_shell(nx_=nx, ny_=ny, n_dir=64, n_fourier=nf, steps=0, rk_tol=1e-8)
    c["cfl"] = cfl
    ref = oracle.run(c, "oracle")
    with grlbm.prepare(c) as r:
        got, st = r.coefficients(), r.stats()
    assert st["rk_nonconverged"] == 0 and st["rk_substeps"] > 0
    for k in COEF:
        assert np.isfinite(got[k]).all(), k
        assert rel_l2(got[k], ref[k]) <= 1e-13, (k, rel_l2(got[k], ref[k]))


@pytest.mark.gpu
def test_a_band_builds_its_own_rows(grlbm, W):
    c = W.curved_shell(nx_=21, ny_=19, n_dir=16, n_fourier=5, steps=0, rk_tol=1e-8)
    with grlbm.prepare(c) as whole, grlbm.prepare(c, rows=(6, 13)) as band:
        a, b = whole.coefficients(), band.coefficients()
    for k in COEF:
        x, y = a[k].reshape(21, 23, 5), b[k].reshape(21, 23, 5)
        assert np.array_equal(x[6:13, 1:-1], y[6:13, 1:-1], equal_nan=True), k
