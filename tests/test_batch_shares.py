"""A batch's concurrent launches on shares (launch shapes below 0): the tiled
forms' grids are cut to their shares, a block then takes many tiles, and the
results are the bits of the problems' own steps."""
import importlib

import numpy as np
import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")

pytestmark = pytest.mark.gpu
FORMS = {"fp32": grlbm.PRECISION_FP32, "fast64": grlbm.FAST_FP64}


def _case(nx, ny, nd, curved=True, moving=False):
    c = W.curved_scatter(nx_=nx, ny_=ny, n_dir=nd, n_fourier=5, steps=4)
    f = c["fields"]
    rng = np.random.default_rng(nx + nd)
    n = f["eta"].size
    f["eta"] = rng.uniform(0.0, 1.0, n)
    if moving:
        f["ux"], f["uy"] = rng.uniform(-0.2, 0.2, n), rng.uniform(-0.2, 0.2, n)
    if not curved:
        c.update(metric_kind=W.MINKOWSKI, streaming_type=W.FLAT_FIXED, excision=-1.0)
    return c


def _kernels(problems, shape):
    """The kernel and grid of each problem's step in a batch step."""
    with grlbm.Batch(problems) as b:
        b.set_shape(shape)
        b.step(1)
    return [r.step_kernel() for r in problems]


@pytest.mark.parametrize("form", ["fp32", "fast64"])
def test_grids_are_cut_to_the_shares(form):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    probs = [grlbm.prepare(_case(248, 240, 32), FORMS[form]) for _ in range(2)]
    try:
        whole = [k["blocks"] for k in _kernels(probs, 0)]
        share = [k["blocks"] for k in _kernels(probs, -1)]
    finally:
        for r in probs:
            r.close()
    assert len(whole) == len(share) == 2
    # two equal problems: half of the resident blocks (at most 8 an SM) each
    assert all(x <= (8 * sms + 1) // 2 for x in share), (whole, share)
    assert all(x < y for x, y in zip(share, whole)), (whole, share)


@pytest.mark.parametrize("shape", [0, -4])
def test_large_problems_keep_the_block_step(shape):
    """A problem that runs the warp-per-tile kernel when it has the GPU to
    itself (512^2 x 16 flat) runs the block step in a batch; the same bits."""
    case = _case(512, 512, 16, curved=False)
    I0 = np.random.default_rng(0).uniform(0.0, 2.0, case["fields"]["eta"].size * 16)
    probs = [grlbm.prepare(case, grlbm.PRECISION_FP32) for _ in range(2)]
    try:
        assert all(k["kernel"] == "block" for k in _kernels(probs, shape))
        probs[0].step(1)
        assert probs[0].step_kernel()["kernel"] == "warp"
        for r in probs:
            r.set_intensity(I0)
        with grlbm.Batch(probs) as b:
            b.set_shape(shape)
            b.step(2)
        got = probs[0].intensity()
        probs[1].set_intensity(I0)
        probs[1].step(2)
        assert np.array_equal(got, probs[1].intensity())
    finally:
        for r in probs:
            r.close()


# grids of many tiles a block, ragged at both edges; every store width and
# both run lengths (200 directions: runs of 4); a moving fluid
@pytest.mark.parametrize("shape", [-1, -2])
@pytest.mark.parametrize("curved", [True, False])
@pytest.mark.parametrize("form", ["fp32", "fast64"])
def test_bits_of_the_own_steps(form, curved, shape):
    cases = [_case(203, 190, 17, curved), _case(150, 211, 34, curved, True), _case(170, 165, 64, curved),
             _case(90, 101, 200, curved)]
    start = [np.random.default_rng(k).uniform(0.0, 2.0, c["fields"]["eta"].size * c["n_dir"]) for k, c in enumerate(cases)]
    want = []
    for c, I0 in zip(cases, start):
        with grlbm.prepare(c, FORMS[form]) as r:
            r.set_intensity(I0)
            r.step(3)
            s = r.stats()
            want.append((r.intensity(), r.moments_if(), s["max_iterations"], s["average_iterations"]))
    probs = [grlbm.prepare(c, FORMS[form]) for c in cases]
    try:
        for r, I0 in zip(probs, start):
            r.set_intensity(I0)
        with grlbm.Batch(probs) as b:
            b.set_shape(shape)
            b.step(3)
        for r, (I, m, most, average) in zip(probs, want):
            assert np.array_equal(r.intensity(), I)
            got = r.moments_if()
            assert all(np.array_equal(got[k], m[k]) for k in m)
            s = r.stats()
            assert s["max_iterations"] == most and s["average_iterations"] == average
    finally:
        for r in probs:
            r.close()
