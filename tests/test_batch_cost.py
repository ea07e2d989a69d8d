"""The forms' costs in the model that shares a batch's launches and deals
replicas, against the step times that they stand for."""
import importlib

import pytest
import torch

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")


def _step_us(case, form):
    with grlbm.prepare(case, form) as r:
        stream = torch.cuda.ExternalStream(r.stream)
        with torch.cuda.stream(stream):
            times = []
            for _ in range(3):
                r.step_async(5)
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(stream)
                r.step_async(20)
                b.record(stream)
                stream.synchronize()
                times.append(a.elapsed_time(b) / 20 * 1e3)
        return min(times)


@pytest.mark.gpu
def test_form_ratios_are_the_measured_ones():
    fixed = W.curved_scatter(nx_=400, ny_=400, n_dir=64, n_fourier=16, steps=1, rk_tol=1e-6)
    adaptive = dict(fixed, streaming_type=W.CURVED_ADAPTIVE)
    base = _step_us(fixed, grlbm.PRECISION_FP32) / grlbm.batch_cost(fixed)
    for case, form in ((fixed, grlbm.FAST_FP64), (fixed, grlbm.PLAIN_FP64), (adaptive, grlbm.PRECISION_FP32),
                       (adaptive, grlbm.PLAIN_FP64)):
        ratio = _step_us(case, form) / grlbm.batch_cost(case, form) / base
        assert 1 / 1.4 < ratio < 1.4, (form, ratio)
