"""GPU: which way a build from edges takes on each side of the rules' lines, with
parity where no other test takes that way."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BUCKETS, LONG_BITS, BITS_4K = 1, 2, 4


def _edges(gb, kind: str, n: int, m: int):
    rng = np.random.default_rng(n)
    if kind == "rmat":
        return gb.gen_rmat(19, 24, seed=5)
    src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
    if kind == "local":
        src = np.arange(m) * n // m
        dst = np.minimum(src + rng.integers(0, 3, m), n - 1)
    if kind == "star":
        src[rng.random(m) < 0.9] = 77
    return src.astype(np.int32), dst.astype(np.int32)


@pytest.mark.parametrize("kind,n,m,flags,buckets", [
    ("uniform", 300_007, 10_600_001, 7, True),
    ("uniform", 300_007, 10_480_000, 7, False),      # fewer than 20 M entries
    ("uniform", 300_007, 21_200_000, 0, True),
    ("uniform", 1 << 22, 10_600_000, 7, True),
    ("uniform", (1 << 22) + 1, 10_600_000, 7, False),
    ("uniform", 300_007, 10_600_001, 7 | 16, False),  # 64-bit row offsets
    ("uniform", 24_000, 10_600_000, 7, True),        # all buckets past shared memory (0.9 M entries)
    ("uniform", 12_500, 10_600_000, 7, False),       # past a bucket's most (1.7 M)
    ("rmat", 1 << 19, 12 << 20, 7, True),
    ("star", 200_000, 10_600_000, 7, False),
    ("local", 1_000_000, 10_600_000, 7, False),
])
def test_buckets(gb, kind, n, m, flags, buckets):
    src, dst = _edges(gb, kind, n, m)
    gb.Graph.from_edges(n, src, dst, flags).close()
    assert bool(gb.lib.gbfs_selftest_build_route() & BUCKETS) == buckets


@pytest.mark.parametrize("n", [24_000, 21 * 1024 + 1])  # 0.9 and 1.01 M entries in each of the full buckets
@pytest.mark.parametrize("flags", [0, 7])
def test_buckets_that_all_overflow_shared_memory(gb, orc, n, flags):
    m = 10_600_000 if flags else 21_200_000
    src, dst = _edges(gb, "uniform", n, m)
    g = gb.Graph.from_edges(n, src, dst, flags)
    assert gb.lib.gbfs_selftest_build_route() & BUCKETS
    row, col = g.csr()
    if flags:
        o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
        want_row, want_col = o.row_offset, o.col_idx
    else:
        key = np.sort(src.astype(np.int64) * n + dst)
        want_row, want_col = np.zeros(n + 1, np.int64), (key % n).astype(np.int32)
        np.cumsum(np.bincount(src, minlength=n), out=want_row[1:])
    assert np.array_equal(row, want_row)
    assert np.array_equal(col, want_col)


RANGE = 32 * 512 * 53  # vertices in the largest range of one CTA


@pytest.mark.parametrize("n,longest,flags,route", [
    (60_000, 2048, 2, 0),
    (60_000, 2049, 2, BITS_4K),
    (60_000, 4096, 2, BITS_4K),
    (60_000, 4097, 2, LONG_BITS),
    (60_000, 4097, 0, 0),  # nothing to deduplicate
    (2 * RANGE, 4096, 2, BITS_4K),
    (2 * RANGE + 1, 4096, 2, 0),
    (5 * RANGE, 4097, 2, LONG_BITS),
    (5 * RANGE + 1, 4097, 2, 0),
])
def test_long_rows(gb, n, longest, flags, route):
    src = np.append(np.full(longest, 7), np.arange(8, 100)).astype(np.int32)
    dst = np.append(np.arange(longest), np.arange(92)).astype(np.int32)
    gb.Graph.from_edges(n, src, dst, flags).close()
    assert gb.lib.gbfs_selftest_build_route() == route
