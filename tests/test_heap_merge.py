"""The warp's merge loop (heap_merge.cuh), run on the CPU as 32-lane arrays with
bounds-checked memory, must leave the parent links of the sequential libstdc++
replay (huffman_build.cuh) on heaps of every shape and tie pattern."""
import ctypes

import numpy as np
import pytest

from helpers import load_selftest

PATTERNS = {
    "all equal": lambda r, n: np.ones(n),
    "ones and twos": lambda r, n: r.integers(1, 3, n),
    "few values": lambda r, n: r.integers(1, 11, n),
    "powers of two": lambda r, n: 1 << r.integers(0, 14, n),
    "log-uniform": lambda r, n: np.exp(r.uniform(0, 11, n)),
    "distinct": lambda r, n: r.permutation(n) + 1,
    "near the limit": lambda r, n: np.maximum(1, (2 ** 31 - 2) // n - r.integers(0, 3, n)),
}


@pytest.mark.parametrize("pattern", sorted(PATTERNS))
def test_warp_merge_matches_sequential_replay(pattern):
    st = load_selftest()
    if st is None:
        pytest.skip("self-test library not built")
    f = st.ccst_heap_merge
    u32p = ctypes.POINTER(ctypes.c_uint32)
    f.argtypes = [u32p, ctypes.c_uint32, ctypes.c_uint32, u32p, u32p]
    rng = np.random.default_rng(5)
    # around every tree depth's edge, odd sizes, and the largest heap
    sizes = list(range(2, 70)) + [127, 128, 129, 255, 256, 257, 1000, 1023, 1024, 1025, 2047, 2048, 4097]
    if pattern in ("few values", "log-uniform"):
        sizes += [8191, 8192, 8193, 12287, 12288]
    for n in sizes:
        p = np.ascontiguousarray(PATTERNS[pattern](rng, n), np.uint32)
        for cap in (256, 1024, 2048, 12288):     # the builders' capacities
            if n > cap or (cap == 12288 and n < 1000 and n % 7):
                continue
            got, want = np.zeros(2 * n, np.uint32), np.zeros(2 * n, np.uint32)
            rc = f(p.ctypes.data_as(u32p), n, cap, got.ctypes.data_as(u32p), want.ctypes.data_as(u32p))
            assert rc == 0, (n, cap)
            assert np.array_equal(got, want), (n, cap)
