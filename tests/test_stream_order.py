"""Set-up work runs on the context's own stream, before the kernels that read
it: that stream does not wait for the default one, where a copy or a memset
may land after the kernels have started."""
import importlib
import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "2dradiation_b200" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_device_memory_is_written_on_a_named_stream(path):
    text = path.read_text()
    assert not re.search(r"\bcudaMemset\s*\(", text)
    for call in re.finditer(r"\bcudaMemcpy\s*\(([^;]*);", text):
        assert "DeviceToHost" in call.group(1), call.group(0)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["PLAIN_FP64", "FAST_FP64", "PRECISION_FP32"])
def test_a_busy_default_stream_changes_nothing(grlbm, W, form):
    """The set-up calls neither wait for the default stream (kept busy for
    a fifth of a second) nor depend on it.  Every node is a source: 300 KB of
    source values, more than a pageable copy passes on by itself."""
    torch = importlib.import_module("torch")
    c = W.curved_scatter(nx_=33, ny_=31, n_dir=32, n_fourier=5, steps=3, rk_tol=1e-6)
    f = c["fields"]
    f["is_initial"][:] = 1
    f["initial_I"] = 0.2 + W.uniform(5, f["eta"].size * 32)
    with grlbm.prepare(c) as r:
        coef = r.coefficients()

    def run(busy):
        with grlbm.Radiation(c, getattr(grlbm, form)) as r:
            for again in range(2):  # (the first pass allocates the sources and records)
                done = torch.cuda.Event()
                if busy and again:
                    torch.cuda._sleep(400_000_000)
                    done.record()
                r.set_fields(f)
                r.set_initial_data(f)
                r.load_initial_data()
                r.set_coefficients(coef)
                if busy and again:
                    assert not done.query()
            r.step(3)
            return [r.intensity()] + list(r.moments_if().values())

    quiet = run(False)
    torch.cuda._sleep(400_000_000)  # the context is created beside it too
    for a, b in zip(quiet, run(True)):
        assert np.array_equal(a, b, equal_nan=True)
    torch.cuda.synchronize()
