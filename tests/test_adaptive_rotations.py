"""The adaptive FP32 step's staged-patch stream against its row-by-row stream
(bands of few rows) from a state whose rotation angles differ from node to
node: both read every corner in that node's previous frame."""
import importlib

import numpy as np
import pytest
import torch

grlbm = importlib.import_module("2dradiation_b200")
W = importlib.import_module("2dradiation_b200.workloads")

pytestmark = pytest.mark.gpu


def _stream(r):
    r.step(1)
    k = r.step_kernel()
    assert k["kernel"] == "adaptive_fp32"
    return "patch" if k["detail"] else "rows"


@pytest.mark.parametrize("nx,ny,nd,nf,cfl", [(161, 85, 33, 5, 0.9), (129, 100, 20, 16, 0.9), (97, 141, 7, 9, 0.9),
                                             (160, 96, 64, 5, 1.8)])
def test_streams_agree_on_rotated_nodes(nx, ny, nd, nf, cfl):
    case = W.curved_scatter(nx_=nx, ny_=ny, n_dir=nd, n_fourier=nf, steps=1)
    case.update(streaming_type=W.CURVED_ADAPTIVE, cfl=cfl)
    n = case["fields"]["eta"].size
    rng = np.random.default_rng(nd)
    case["fields"]["eta"] = rng.uniform(0.0, 0.1, n)
    # a beam at every node, in a direction of its own
    phi = (np.arange(nd) + 0.5) * (2 * np.pi / nd)
    I0 = np.exp(2.0 * np.cos(phi[None, :] - rng.uniform(0.0, 2 * np.pi, n)[:, None]))
    rows = ny + 2
    with grlbm.prepare(case, grlbm.PRECISION_FP32) as r:
        r.set_intensity(I0)
        r.step(2)
        state = [torch.empty(rows * b, dtype=torch.uint8, device="cuda")
                 for b in (r.row_bytes(), r.node_row_bytes(grlbm.ROWS_ANGLES), r.node_row_bytes(grlbm.ROWS_MOMENTS))]

        def copy(q, to_buffer):
            q.copy_rows(0, rows, state[0].data_ptr(), to_buffer)
            q.copy_node_rows(grlbm.ROWS_ANGLES, 0, rows, state[1].data_ptr(), to_buffer)
            q.copy_node_rows(grlbm.ROWS_MOMENTS, 0, rows, state[2].data_ptr(), to_buffer)
            q.sync()

        torch.cuda.synchronize()
        copy(r, True)
        angles = state[1].cpu().numpy().view(np.float64).reshape(rows, nx + 2)[1:-1, 1:-1]
        assert np.count_nonzero(angles) > 0.8 * angles.size
        assert np.mean(np.abs(np.diff(angles, axis=0)) > 1e-3) > 0.8 and np.mean(np.abs(np.diff(angles, axis=1)) > 1e-3) > 0.8
        assert _stream(r) == "patch"
        whole, whole_I = r.moments_if(), r.intensity().reshape(n, nd)
    nodes = np.arange(n).reshape(rows, nx + 2)
    for lo in range(1, ny + 1, 30):
        hi = min(lo + 30, ny + 1)
        with grlbm.prepare(case, grlbm.PRECISION_FP32) as r:
            r.set_rows(lo, hi)
            r.set_intensity(I0)  # excised nodes keep theirs in both buffers
            copy(r, False)
            assert _stream(r) == "rows"
            band, band_I = r.moments_if(), r.intensity().reshape(n, nd)
        at = nodes[lo:hi, 1 : nx + 1]
        assert np.array_equal(whole_I[at], band_I[at]), lo
        for k in whole:
            assert np.array_equal(whole[k][at], band[k][at]), (k, lo)
