"""GPU parity of the CSR build's per-row sorts at the edges of their length
classes: warp, CTA, and rows in chunks of 4096 merged 0 to 4 times."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = (1, 2, 7, 8, 9, 10, 15, 16, 17, 31, 32, 33, 8, 16, 12, 63, 64, 65, 128, 129, 512, 513, 1024, 1025, 2048, 2049, 4095, 4096, 4097, 8191, 8192, 8193, 12_289,
           16_384, 16_385, 40_000, 70_001)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("values", ["distinct", "repeated", "few", "last_chunk_equal"])
@pytest.mark.parametrize("dedup", [False, True])
def test_sorted_rows_of_every_length(gb, orc, dedup, values, wide):
    rng = np.random.default_rng(len(values) + dedup)
    n = 100_000
    src, dst = [], []
    for r, d in enumerate(LENGTHS):
        if values == "distinct":
            v = rng.choice(n, d, replace=False)
        elif values == "repeated":
            v = rng.integers(0, max(1, d // 2), d)
        elif values == "few":
            v = rng.integers(n - 3, n, d)  # the largest ids among them
        else:
            v = np.where(np.arange(d) < 4000, rng.integers(0, n, d), 77)
        src.append(np.full(d, 3 * r + 1))
        dst.append(v)
    src, dst = np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)
    p = rng.permutation(len(src))
    src, dst = np.ascontiguousarray(src[p]), np.ascontiguousarray(dst[p])
    g = gb.Graph.from_edges(n, src, dst, (gb.DEDUP if dedup else 0) | (gb.WIDE_ROWS if wide else 0))
    o = orc.csr_build(n, src, dst, orc.DEDUP if dedup else 0)
    row, col = g.csr()
    assert np.array_equal(row, o.row_offset)
    want = o.col_idx.copy()  # in file order without deduplication
    for r in range(0, 3 * len(LENGTHS)):
        want[row[r]:row[r + 1]].sort()
    assert np.array_equal(col, want)
