"""The page-locked buffers of the read-back: shared, bounded, per device, and
never handed out again after a reset of the device has freed them, so that a
caller may reset it between contexts."""
import os
import shutil
import subprocess
import sys
import threading
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_buffers_are_bounded_and_do_not_survive_a_reset(tmp_path):
    exe = tmp_path / "check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(HERE.parent / "2dradiation_b200" / "csrc"), "-o",
                    str(exe), str(HERE / "read_back_buffers_check.cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout


@pytest.mark.gpu
def test_contexts_after_others_and_threads_read_the_same(grlbm, W):
    """Contexts one after another, and several read from threads at once:
    each gets its own values."""
    case = W.curved_shell(nx_=61, ny_=50, n_dir=16, n_fourier=5, steps=2)
    want = []
    for k in range(3):
        with grlbm.prepare(case, grlbm.PRECISION_FP32) as r:
            r.step(2 + k)
            want.append([r.intensity()] + list(r.moments_if().values()))
    rads = [grlbm.prepare(case, grlbm.PRECISION_FP32) for _ in range(6)]
    got = [None] * len(rads)

    def work(k):
        rads[k].step(2 + k % 3)
        got[k] = [rads[k].intensity()] + list(rads[k].moments_if().values())

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(rads))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in rads:
        r.close()
    for k, out in enumerate(got):
        for a, b in zip(out, want[k % 3]):
            assert np.array_equal(a, b, equal_nan=True)


RESET = """
import ctypes, importlib, sys
import numpy as np
grlbm = importlib.import_module("2dradiation_b200")
case = grlbm.workloads.flat_beam(nx_=40, ny_=40, n_dir=8, steps=5)

def moments():
    with grlbm.prepare(case) as r:
        r.step(5)
        return r.moments_if()

first = moments()
rt = ctypes.CDLL(sys.argv[1])
assert rt.cudaDeviceReset() == 0
keep = []
for _ in range(8):  # what the reset freed may be page-locked again by others
    p = ctypes.c_void_p()
    assert rt.cudaHostAlloc(ctypes.byref(p), ctypes.c_size_t(1 << 20), 0) == 0
    ctypes.memset(p, 0x5A, 1 << 20)
    keep.append(p)
again = moments()
assert all(np.array_equal(first[k], again[k]) for k in first)
assert all(ctypes.string_at(p, 1 << 20) == b"\\x5a" * (1 << 20) for p in keep)
print("ok")
"""


@pytest.mark.gpu
def test_a_device_reset_between_contexts(tmp_path):
    """The caller resets the device when no context is left (in a process of
    its own: the reset ends that process's CUDA context only)."""
    torch = pytest.importorskip("torch")
    libs = sorted(Path(torch.__file__).parents[1].glob("nvidia/cuda_runtime/lib/libcudart.so.*"))
    if not libs:
        pytest.skip("no CUDA runtime library to reset the device through")
    script = tmp_path / "reset.py"
    script.write_text(RESET)
    out = subprocess.run([sys.executable, str(script), str(libs[0])], cwd=HERE.parent, capture_output=True, text=True,
                         timeout=300, env=dict(os.environ, PYTHONPATH=str(HERE.parent)))
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stderr[-2000:]
