"""Results reach pageable memory through the context's page-locked halves and
page-locked memory directly: the same values, with some outputs left out, at
grids of less than a half, of several, and of a ragged last one."""
import ctypes
import importlib

import numpy as np
import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")
KEYS = ("E", "Fx", "Fy", "Pxx", "Pxy", "Pyy")


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["PLAIN_FP64", "FAST_FP64", "PRECISION_FP32"])
@pytest.mark.parametrize("nx,ny", [(5, 3), (104, 103), (211, 180)])
def test_pageable_and_page_locked_read_backs_agree(nx, ny, form):
    torch = importlib.import_module("torch")
    case = W.curved_shell(nx_=nx, ny_=ny, n_dir=8, n_fourier=5, steps=3)
    with grlbm.prepare(case, getattr(grlbm, form)) as r:
        r.step(3)
        m, I = r.moments_if(), r.intensity()
        pinned = [torch.full((r.nxy,), -1.0, dtype=torch.float64, pin_memory=True) for _ in KEYS]
        ptr = lambda t: ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))
        f = grlbm.lib().grlbm_get_moments_if
        assert f(r.h, *[ptr(t) for t in pinned]) == 0
        for k, t in zip(KEYS, pinned):
            assert np.array_equal(m[k], t.numpy(), equal_nan=True)
        some = {k: np.full(r.nxy, -1.0) for k in KEYS}
        args = [some[k].ctypes.data_as(ctypes.POINTER(ctypes.c_double)) if k in ("Fx", "Pyy") else None for k in KEYS]
        assert f(r.h, *args) == 0
        for k in KEYS:
            assert np.array_equal(some[k], m[k] if k in ("Fx", "Pyy") else np.full(r.nxy, -1.0), equal_nan=True)
        out = torch.empty(r.nxy * r.nd, dtype=torch.float64, pin_memory=True)
        assert grlbm.lib().grlbm_get_intensity(r.h, ptr(out)) == 0
        assert np.array_equal(I, out.numpy(), equal_nan=True)
