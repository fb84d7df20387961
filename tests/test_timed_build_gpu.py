"""The timed build times the build: for clouds that are not built in one launch its
steps add up to what the build takes, and steps that the build does not have take
nothing."""
import ctypes as C
import statistics

import pytest
import torch

pytestmark = pytest.mark.gpu


def steps_us(b, pts, n):
    from pipeline_gb300 import _lib

    lib = b.lib
    count = lib.oct_build_step_count()
    names = [lib.oct_build_step_name(k).decode() for k in range(count)]
    stream = torch.cuda.current_stream()
    rows = []
    for _ in range(12):
        events = [torch.cuda.Event(enable_timing=True) for _ in range(count)]
        for e in events:
            e.record(stream)
        torch.cuda.synchronize()
        handles = (C.c_void_p * count)(*[e.cuda_event for e in events])
        _lib.check(lib.oct_build_octree_timed(
            pts.data_ptr(), n, 0.0, 1024.0, C.byref(b._out), b.workspace.data_ptr(),
            b.workspace.numel(), handles, count, stream.cuda_stream), "oct_build_octree_timed")
        torch.cuda.synchronize()
        rows.append([events[k - 1].elapsed_time(events[k]) * 1e3 for k in range(1, count)])
    return {name: statistics.median(r[k] for r in rows) for k, name in enumerate(names[1:])}


# sizes of the one-launch sort, of the MSD form, and of the passes past it
@pytest.mark.parametrize("n", [2_500_000, 6_000_000, 17_000_000])
def test_steps_add_up_to_the_build(n):
    """Within a seventh: thirteen events, and single builds (no launch hides behind
    another build) against builds in a row."""
    from pipeline_gb300.pipeline import OctreeBuilder

    g = torch.Generator(device="cuda").manual_seed(1)
    pts = torch.rand((n, 4), generator=g, device="cuda") * 1023.9
    b = OctreeBuilder(n)
    b.build(pts, 0.0, 1024.0)
    want = b.result()["oct_nodes"].tobytes()
    a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    build = 1e30
    for _ in range(5):
        torch.cuda.synchronize()
        a.record()
        for _ in range(10):
            b.build(pts, 0.0, 1024.0)
        e.record()
        e.synchronize()
        build = min(build, a.elapsed_time(e) * 100)
    steps = steps_us(b, pts, n)
    assert b.result()["oct_nodes"].tobytes() == want
    total = sum(steps.values())
    assert 6 / 7 * build < total < 8 / 7 * build, (build, steps)
    if n < 4_000_000:
        absent = ("histogram scan", "sort pass 1", "sort pass 2", "msd buckets")
        assert all(steps[k] < 3 for k in absent), steps
