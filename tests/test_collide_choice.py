"""Which kernel the plain form's collide runs: the cells' streamed values in a
column of shared memory up to 91 directions.  The bits against the oracle are test_plain_paths.py's."""
import importlib
import json
import re

import pytest

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")


def _column(r, path):
    """Whether the collide that a step launches has the column."""
    from torch.profiler import ProfilerActivity, profile
    r.step(1)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        r.step(1)
    p.export_chrome_trace(str(path))
    names = [e["name"] for e in json.loads(path.read_text())["traceEvents"]
             if e.get("cat") == "kernel" and "k_collide_plain" in e["name"]]
    assert len(names) == 1, names
    flags = re.search(r"k_collide_plain<(.*?)>", names[0])[1].split(", ")
    return flags[2] == "true"


@pytest.mark.gpu
@pytest.mark.parametrize("nd", [32, 90, 91, 92])
@pytest.mark.parametrize("adaptive", [False, True])
def test_column_by_directions(nd, adaptive, tmp_path):
    case = W.curved_scatter(nx_=20, ny_=17, n_dir=nd, n_fourier=3, steps=1, rk_tol=1e-6)
    case.update(metric_kind=W.MINKOWSKI, streaming_type=W.FLAT_ADAPTIVE if adaptive else W.FLAT_FIXED, excision=-1.0)
    with grlbm.prepare(case, grlbm.PLAIN_FP64) as r:
        assert _column(r, tmp_path / "a.json") == (nd <= 91)
