"""What the sorts that take the place of digit passes cost where keys are uneven: no
more than the passes, which another sort configuration selects, by a margin for
the clock (each fault that this is held against was 1.2 times and more)."""
import contextlib
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
MARGIN = 1.12


@contextlib.contextmanager
def passes():
    """Plans and sorts of this block take digit passes."""
    from pipeline_gb300 import _lib

    lib, old = _lib.load(), (ctypes.c_int * 4)()
    lib.oct_get_sort_config(old)
    assert lib.oct_set_sort_config(10, 16, 24, 1) == 0
    try:
        yield
    finally:
        assert lib.oct_set_sort_config(*list(old)) == 0


def points(codes):
    pts = torch.ones((codes.numel(), 4), device="cuda")
    for axis in range(3):
        cell = torch.zeros_like(codes)
        for bit in range(10):
            cell |= ((codes >> (3 * bit + axis)) & 1) << bit
        pts[:, axis] = cell + 0.5
    return pts


def codes(kind, n, seed=1):
    g = torch.Generator(device="cuda").manual_seed(seed)
    some = lambda span: torch.randint(0, span, (n,), generator=g, device="cuda")  # noqa: E731
    even, low = some(1 << 30), 123_456_789
    share = torch.rand(n, generator=g, device="cuda")
    if kind == "one bucket":
        return (5 << 20) + some(1 << 20)
    if kind == "one value":
        return torch.full_like(even, low)
    if kind == "even":
        return even
    if kind == "lumps":  # even at the top, not below
        return (some(4096) << 18) + some(600)
    few = {"nine tenths": lambda: low, "ten values": lambda: some(10) * 100_000_007,
           "narrow": lambda: low + some(1 << 12)}[kind]()
    return torch.where(share < 0.9, few, even)


def best_us(run, reps):
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = 1e30
    for _ in range(6):
        torch.cuda.synchronize()
        a.record()
        for _ in range(reps):
            run()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) / reps * 1e3)
    return best


@pytest.mark.parametrize("kind", ["one bucket", "one value", "narrow"])
@pytest.mark.parametrize("clouds,n", [(64, 49_152), (16, 30_000), (64, 12_288)])
def test_batched_builds_of_concentrated_clouds(kind, clouds, n):
    from pipeline_gb300.batch import BatchOctreeBuilder

    pts = torch.cat([points(codes(kind, n, c)) for c in range(clouds)])
    lows = torch.zeros(clouds, device="cuda")
    extents = torch.full((clouds,), 1024.0, device="cuda")

    def us():
        b = BatchOctreeBuilder([n] * clouds)
        return best_us(lambda: b.build(pts, lows, extents), 10)

    with passes():
        want = us()
    assert us() < MARGIN * want


def sort_us(src, bits):
    from pipeline_gb300.kernels import k_SimpleRadixSort

    keys, alt = torch.empty_like(src), torch.empty_like(src)

    def run():
        keys.copy_(src)
        k_SimpleRadixSort(keys, alt, src.numel(), key_bits=bits)

    return best_us(run, 10)


@pytest.mark.parametrize("kind", ["nine tenths", "ten values", "narrow", "lumps"])
@pytest.mark.parametrize("n", [1_000_000, 3_900_000, 4_100_000, 8_000_000])
def test_sorts_of_keys_of_a_few_values(kind, n):
    src = codes(kind, n).to(torch.int32)
    for bits in (30, 32):
        with passes():
            want = sort_us(src, bits)
        assert sort_us(src, bits) < MARGIN * want


@pytest.mark.parametrize("kind", ["even", "nine tenths", "ten values", "narrow", "one bucket",
                                  "one value", "lumps"])
@pytest.mark.parametrize("n", [(1 << 21) + 1, 4_000_000, 4_000_001, 1 << 23, (1 << 23) + 1])
def test_few_values_sort_like_torch(kind, n):
    """On both sides of the array sizes from which the keys are looked at first, may be
    left to passes, and take passes alone; with bits above key_bits as well."""
    from pipeline_gb300.kernels import k_SimpleRadixSort

    src = codes(kind, n).to(torch.int32)
    for bits, above in ((30, 0), (32, 0), (30, 1 << 30)):
        keys = src + above
        want = torch.sort(keys).values
        alt, status = torch.empty_like(keys), torch.zeros(1, dtype=torch.int32, device="cuda")
        k_SimpleRadixSort(keys, alt, n, key_bits=bits, status=status)
        assert int(status[0]) == 0 and torch.equal(keys, want)


def narrow(kind, n, bits):
    g = torch.Generator(device="cuda").manual_seed(4)
    some = torch.randint(0, 1 << bits, (n,), generator=g, device="cuda")
    share = torch.rand(n, generator=g, device="cuda")
    part = {"even": 0.0, "half": 0.5, "nine tenths": 0.9, "one value": 1.0}[kind]
    return torch.where(share < part, torch.full_like(some, 3), some).to(torch.int32)


@pytest.mark.parametrize("bits", [4, 8, 10, 11, 16, 20])
@pytest.mark.parametrize("kind", ["even", "half", "nine tenths", "one value"])
def test_sorts_of_narrow_keys(kind, bits):
    """One and two digit passes are little to be faster than: sizes on both sides of a
    cluster's, of the first look's, and near the largest array of one launch."""
    from pipeline_gb300.kernels import k_SimpleRadixSort

    for n in (8192, 8193, 16_000, 130_000, 1 << 20, (1 << 20) + 1, 1_800_000, 3_900_000):
        src = narrow(kind, n, bits)
        keys, alt = src.clone(), torch.empty_like(src)
        k_SimpleRadixSort(keys, alt, n, key_bits=bits)
        assert torch.equal(keys, torch.sort(src).values)
        with passes():
            want = sort_us(src, bits)
        assert sort_us(src, bits) < MARGIN * want, n


def build_us(pts):
    from pipeline_gb300.pipeline import OctreeBuilder

    b = OctreeBuilder(pts.shape[0])
    return best_us(lambda: b.build(pts, 0.0, 1024.0), 10)


@pytest.mark.parametrize("kind", ["two values", "one octant"])
@pytest.mark.parametrize("n", [4_300_000, 8_300_000, 16_700_000])
def test_builds_of_clouds_that_the_msd_form_refuses(kind, n):
    g = torch.Generator(device="cuda").manual_seed(2)
    c = torch.randint(0, 1 << 30, (n,), generator=g, device="cuda")
    if kind == "two values":
        share = torch.rand(n, generator=g, device="cuda")
        c = torch.where(share < 0.45, 123_456_789, torch.where(share < 0.9, 987_654_321, c))
    else:
        c = (9 << 18) + c % (1 << 18)
    pts = points(c)
    del c
    with passes():
        want = build_us(pts)
    assert build_us(pts) < MARGIN * want


@pytest.mark.parametrize("kind,most", [("even", 0.9), ("nine tenths", MARGIN), ("lumps", 0.9)])
@pytest.mark.parametrize("n", [4_000_001, (1 << 22) - 1])
def test_builds_up_to_the_msd_size_take_one_sort(kind, most, n):
    """Between the sizes from which sorts alone may take passes and builds the MSD form."""
    from pipeline_gb300.pipeline import OctreeBuilder

    pts = points(codes(kind, n))

    def nodes():
        b = OctreeBuilder(n)
        b.build(pts, 0.0, 1024.0)
        return b.result()["oct_nodes"].tobytes()

    with passes():
        want, tree = build_us(pts), nodes()
    assert nodes() == tree
    assert build_us(pts) < most * want


@pytest.mark.parametrize("kind", ["nine tenths", "one bucket"])
@pytest.mark.parametrize("n", [1_000_000, 8_300_000, 16_700_000])
def test_learned_builds_whose_model_does_not_fit(kind, n):
    """The fall-back runs, and costs no more than by passes; the tree is the plain build's."""
    from pipeline_gb300.learned import LearnedCDF
    from pipeline_gb300.pipeline import LearnedOctreeBuilder, OctreeBuilder

    g = torch.Generator(device="cuda").manual_seed(4)
    other = torch.randint(0, 1 << 30, (100_000,), generator=g, device="cuda").to(torch.int32)
    model = LearnedCDF(1024).fit(other, n_segments=1024, steps=20, n_buckets=4096)
    pts = points(codes(kind, n))

    def built():
        b = LearnedOctreeBuilder(n, model)
        us = best_us(lambda: b.build(pts, 0.0, 1024.0), 10)
        return us, b

    with passes():
        want, _ = built()
    got, b = built()
    assert b.lsort_stats()["fallback"] == 1
    assert got < MARGIN * want
    result = b.result()
    del b
    plain = OctreeBuilder(n)
    plain.build(pts, 0.0, 1024.0)
    want = plain.result()
    assert result["status"] == want["status"] == 0
    for key in ("sorted_unique", "parent", "prefix_sum", "oct_nodes"):
        assert result[key].tobytes() == want[key].tobytes(), key


def test_sort_that_may_be_left_to_passes_replayed_from_a_graph():
    """One graph over keys that the one-launch sort takes, leaves after the look, and
    leaves after its count (bits above key_bits in keys that look even)."""
    from pipeline_gb300.kernels import k_SimpleRadixSort

    n = 4_500_001
    src = torch.zeros(n, dtype=torch.int32, device="cuda")
    keys, alt = torch.empty_like(src), torch.empty_like(src)
    k_SimpleRadixSort(keys.zero_(), alt, n, key_bits=30)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        keys.copy_(src)
        k_SimpleRadixSort(keys, alt, n, key_bits=30)
    for kind, above in (("even", 0), ("narrow", 0), ("even", 1 << 30), ("one value", 0), ("even", 0)):
        src.copy_(codes(kind, n).to(torch.int32) + above)
        graph.replay()
        assert torch.equal(keys, torch.sort(src).values), (kind, above)


@pytest.mark.parametrize("digits", [False, True])
@pytest.mark.parametrize("n", [100_001, 4_100_003])
def test_lsort_fall_back_sorts_the_keys_in_place(n, digits):
    """As the header promises, whichever sort the fall-back takes."""
    from pipeline_gb300.learned import LearnedCDF
    from pipeline_gb300.pipeline import lsort_unique

    g = torch.Generator(device="cuda").manual_seed(6)
    other = torch.randint(0, 1 << 30, (100_000,), generator=g, device="cuda").to(torch.int32)
    model = LearnedCDF(1024).fit(other, n_segments=1024, steps=20, n_buckets=1024)
    for kind in ("narrow", "one bucket"):
        keys = codes(kind, n).to(torch.int32)
        want = torch.sort(keys).values
        with passes() if digits else contextlib.nullcontext():
            unique, stats = lsort_unique(keys, model)
        assert stats["fallback"] == 1
        assert torch.equal(keys, want) and torch.equal(unique, torch.unique_consecutive(want))
