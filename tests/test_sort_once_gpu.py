"""The one-launch sort against NumPy and against the digit passes (which another
sort configuration selects): sizes around a warp, a CTA's least share, one
cluster, a CTA's registers and several tiles per CTA; keys that are even, in
few buckets (split by further bits), in few values (counted), almost all equal
(digit passes inside the launch), or with bits above key_bits."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [2, 33, 1023, 1025, 8192, 8193, 200_001, 152 * 16384, 152 * 16384 + 1, 3_000_017]


def make(kind, n, bits, rng):
    a = rng.integers(0, 1 << bits, n, dtype=np.uint64)
    if kind == "clustered":  # dense around few centres, some noise
        c = rng.integers(0, 1 << bits, 24, dtype=np.uint64)
        width = (1 << np.arange(24) % bits).astype(np.uint64)
        p = rng.integers(0, 24, n)
        near = c[p] + rng.integers(0, 1 << 62, n, dtype=np.uint64) % width[p]
        a = np.where(rng.random(n) < 0.05, a, near)
    elif kind == "one bucket":
        a = a % (1 << max(bits - 12, 1))
    elif kind == "frequent":  # a few values that hold 4% each
        a = np.where(rng.random(n) < 0.2, a[rng.integers(0, 5, n) % n], a)
    elif kind == "equal":
        a = np.where(rng.random(n) < 0.99, a[0], a)
    elif kind == "falling":
        a = np.sort(a)[::-1]
    elif kind == "high bits":
        a = rng.integers(0, 1 << 32, n, dtype=np.uint64)
        return a.astype(np.uint32)
    return (a % (1 << bits)).astype(np.uint32)


def run(a, bits, shift=0):
    from pipeline_gb300.kernels import k_SimpleRadixSort

    store = torch.zeros(len(a) + shift, dtype=torch.int32, device="cuda")
    keys = store[shift:]
    keys.copy_(torch.from_numpy(a.view(np.int32)))
    alt = torch.empty(len(a) + shift, dtype=torch.int32, device="cuda")[shift:]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    k_SimpleRadixSort(keys, alt, len(a), key_bits=bits, status=status)
    assert int(status[0]) == 0
    return keys.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("kind", ["even", "clustered", "one bucket", "frequent", "equal",
                                  "falling"])
def test_sorts_like_numpy(kind):
    rng = np.random.default_rng(len(kind))
    for n in SIZES:
        for bits in (30, 32) + ((1, 11, 13, 17) if n in (8193, 152 * 16384 + 1) else ()):
            a = make(kind, n, bits, rng)
            got = run(a, bits, shift=n & 1)
            assert got.tobytes() == np.sort(a).tobytes(), (kind, n, bits)


@pytest.mark.parametrize("kind", ["high bits", "clustered"])
def test_same_as_the_digit_passes(kind):
    from pipeline_gb300 import _lib

    lib = _lib.load()
    old = (ctypes.c_int * 4)()
    lib.oct_get_sort_config(old)
    rng = np.random.default_rng(3)
    for n in (77, 8192, 8193, 500_003, 2_600_001):
        for bits in (9, 20, 25, 30):
            a = make(kind, n, bits, rng)
            got = run(a, bits)
            try:
                assert lib.oct_set_sort_config(10, 16, 24, 1) == 0
                want = run(a, bits)
            finally:
                lib.oct_set_sort_config(*list(old))
            # (keys alike in the bits that order them may lie in any order: the
            # passes' first digit is ranked by atomics)
            low = np.uint32((1 << 10 * -(-bits // 10)) - 1)
            assert (got & low).tobytes() == (want & low).tobytes(), (kind, n, bits)
            assert np.sort(got).tobytes() == np.sort(want).tobytes(), (kind, n, bits)


def test_replayed_from_a_graph():
    from pipeline_gb300.kernels import k_SimpleRadixSort

    n = 700_001
    rng = np.random.default_rng(4)
    src = torch.zeros(n, dtype=torch.int32, device="cuda")
    keys, alt = torch.empty_like(src), torch.empty_like(src)
    k_SimpleRadixSort(keys.zero_(), alt, n)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        keys.copy_(src)
        k_SimpleRadixSort(keys, alt, n)
    for kind in ("even", "equal", "clustered", "even"):
        a = make(kind, n, 32, rng)
        src.copy_(torch.from_numpy(a.view(np.int32)))
        g.replay()
        assert keys.cpu().numpy().view(np.uint32).tobytes() == np.sort(a).tobytes(), kind
