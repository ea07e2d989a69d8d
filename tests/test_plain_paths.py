"""The plain form's two kernels at the edges of their shapes: the staged
stream's blocks (16 x 4 cells; up to 57, up to 88 and more directions) and the
collide's column (up to 90 directions), its passes for a fluid at rest with and
without anisotropic scattering, and its shortcuts -- each bit for bit against
the oracle from the oracle's own tables."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.parametrize("nd", range(4, 257))
def test_consecutive_rows_start_at_most_one_direction_apart(grlbm, nd):
    """The stream reads the 5 directions from a row's first one on for the
    row and the next: both rows are consecutive directions, the second
    starting at the same direction or the next."""
    idx = np.zeros(40 * nd, dtype=np.int64)
    rc = grlbm.lib().grlbm_host_stencil(nd, 1, None, None, None, None, idx.ctypes.data_as(C.POINTER(C.c_int64)), None)
    assert rc == 0
    idx = idx.reshape(-1, 4)
    assert np.array_equal(idx, (idx[:, :1] + np.arange(4)) % nd)
    shift = (np.roll(idx[:, 0], -1) - idx[:, 0]) % nd
    assert shift.max() <= 1


def problem(W, fluid, nx, ny, nd, cfl):
    c = W.curved_scatter(nx_=nx, ny_=ny, n_dir=nd, n_fourier=5, steps=3, rk_tol=1e-6)
    c["cfl"] = cfl
    f = c["fields"]
    n = f["eta"].size
    u = W.uniform(21, n * (nd + 1)).reshape(n, nd + 1)
    f["is_initial"][:] = 1
    I = 0.2 + u[:, :nd]
    if fluid == "extremes":  # tiny, zero and ordinary intensities side by side
        I *= np.choose((u[:, nd] * 3).astype(int), [1e-290, 0.0, 1.0])[:, None]
    f["initial_I"] = I.reshape(-1)
    if fluid in ("absorb", "vacuum"):
        f["kappa0"][:] = 0.0
    if fluid == "vacuum":
        f["kappaA"][:] = np.where(u[:, nd] < 0.2, 0.3, 0.0)
        f["eta"][:] = np.where(u[:, nd] > 0.9, 0.5, 0.0)
    if fluid == "aniso":
        f["kappa1"][:] = 0.3 * u[:, nd]
    if fluid == "sink":  # negative emission: sources of either sign
        f["eta"][:] = u[:, nd] - 0.5
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("fluid,nx,ny,nd,cfl", [
    ("scatter", 19, 23, 5, 0.9), ("absorb", 16, 4, 20, 0.9), ("vacuum", 33, 9, 32, 0.9), ("aniso", 17, 19, 57, 0.9),
    ("scatter", 15, 21, 58, 0.9), ("vacuum", 18, 7, 88, 0.9), ("absorb", 21, 10, 89, 0.9), ("scatter", 16, 9, 90, 0.9),
    ("aniso", 20, 6, 91, 0.9), ("extremes", 31, 13, 24, 0.9), ("sink", 20, 13, 33, 0.9)])
def test_plain_step_bit_for_bit(grlbm, W, oracle, fluid, nx, ny, nd, cfl):
    c = problem(W, fluid, nx, ny, nd, cfl)
    ref = oracle.run(c, "oracle")
    with grlbm.Radiation(c) as r:
        r.set_fields(c["fields"])
        r.set_initial_data(c["fields"])
        r.load_initial_data()
        r.set_coefficients(ref)
        r.step(int(c["n_steps"]))
        got = dict(r.moments_if(), I=r.intensity())
        st = r.stats()
    for k in ("E", "Fx", "Fy", "Pxx", "Pxy", "Pyy", "I"):
        assert np.array_equal(got[k], ref[k], equal_nan=True), k
    assert st["max_iterations"] == ref["max_iterations"]
    assert st["average_iterations"] == pytest.approx(ref["average_iterations"], rel=1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("nd,cfl", [(36, 1.5), (70, 2.3)])
def test_staged_stream_equals_the_gather_from_global_memory(grlbm, W, monkeypatch, nd, cfl):
    """Departures more than a cell away leave the staged patch: the same bits
    as the general gather (which 64-bit offsets select)."""
    c = problem(W, "scatter", 22, 18, nd, cfl)
    got = []
    for wide in ("0", "1"):
        monkeypatch.setenv("GRLBM_WIDE_OFFSETS", wide)
        with grlbm.prepare(c) as r:
            r.step(3)
            got.append(dict(r.moments_if(), I=r.intensity()))
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k], equal_nan=True), k
