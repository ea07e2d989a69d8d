"""A read-back moves the arrays that are asked for and no others."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_only_wanted_arrays_are_moved(tmp_path):
    exe = tmp_path / "check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(HERE.parent / "2dradiation_b200" / "csrc"), "-o", str(exe),
                    str(HERE / "read_back_plan_check.cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
    capi = (HERE.parent / "2dradiation_b200" / "csrc" / "grlbm_capi.cu").read_text()
    assert "ReadBackPlan plan(dst, nq, per" in capi  # the read-back follows it
