"""The grid barriers of the one-launch build and the one-launch sort when a block
never comes: every wait ends within its bound, the status says so, and the counts
of an earlier build are gone."""
import ctypes as C
import time

import pytest
import torch

from oracle import oracle as O
from pipeline_gb300 import _lib

pytestmark = pytest.mark.gpu
LIMIT_NS = 2_000_000


def test_build_reports_a_barrier_that_nobody_completes():
    from pipeline_gb300.pipeline import OctreeBuilder

    lib, n = _lib.load(), 50_000
    pts = O.init_random_vec4(n, seed=6)
    d = torch.from_numpy(pts).cuda()
    b = OctreeBuilder(n, 64)  # too few nodes: counts and a status bit of its own are left behind
    b.build(d, 0.0, 1024.0)
    torch.cuda.synchronize()
    left = b.d_counts.tolist()
    assert left[0] > 0 and left[2] > 64 and left[3] == _lib.OCT_STATUS_CAPACITY
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    t0 = time.perf_counter()
    _lib.check(lib.oct_diag_build_timeout(d.data_ptr(), n, 0.0, 1024.0, C.byref(b._out), LIMIT_NS,
                                          b.workspace.data_ptr(), b.workspace.numel(), s), "diag")
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 < 0.5
    assert b.d_counts.tolist() == [0, 0, 0, _lib.OCT_STATUS_SPIN_TIMEOUT]
    host = (C.c_int32 * 4)()
    assert lib.oct_read_counts(b.d_counts.data_ptr(), host, s) == _lib.OCT_ERR_DEVICE
    b = OctreeBuilder(n)
    b.build(d, 0.0, 1024.0)
    got = b.result()
    assert got["status"] == 0
    assert got["oct_nodes"].tobytes() == O.build_all(pts, 0.0, 1024.0)["oct_nodes"].tobytes()


def test_sort_reports_a_barrier_that_nobody_completes():
    lib = _lib.load()
    ws = torch.empty(lib.oct_diag_wait_workspace_bytes(), dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    args = (_lib.OCT_DIAG_WAIT_GRID, LIMIT_NS, ws.data_ptr())
    assert lib.oct_diag_lookback_timeout(*args, 8192, status.data_ptr(), s) == _lib.OCT_ERR_WORKSPACE
    t0 = time.perf_counter()
    _lib.check(lib.oct_diag_lookback_timeout(*args, ws.numel(), status.data_ptr(), s), "diag")
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 < 0.5
    assert int(status.item()) == _lib.OCT_STATUS_SPIN_TIMEOUT


@pytest.mark.parametrize("n", [0, 1, 8192, 1 << 30])
def test_build_diagnosis_takes_cooperative_builds_only(n):
    out = _lib.OctBuildOutputs()
    assert _lib.load().oct_diag_build_timeout(None, n, 0.0, 1.0, C.byref(out), LIMIT_NS, None, 0,
                                              None) == _lib.OCT_ERR_INVALID_ARG
