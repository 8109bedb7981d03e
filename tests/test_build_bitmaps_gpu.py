"""GPU parity of the CSR build's long rows through bitmaps of the vertices, at the
sizes where another CTA joins a row's cluster and where rows leave the path."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RANGE = 32 * 512 * 53  # vertices in the largest range of one CTA
LENGTHS = (2048, 2049, 4096, 4097, 9000, 4097, 60_001, 33)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n", [60_002, RANGE, RANGE + 1, 2 * RANGE, 2 * RANGE + 1, 3 * RANGE + 5, 5 * RANGE, 5 * RANGE + 1])
def test_long_rows(gb, orc, n, wide):
    rng = np.random.default_rng(n)
    src, dst = [], []
    for r, d in enumerate(LENGTHS):
        v = rng.integers(0, n, d)
        edges = np.arange(0, n, 16 * 32)  # borders of words, threads and ranges
        edges = np.concatenate([edges, edges[1:] - 1, [n - 1]])
        k = min(d // 2, len(edges))
        v[:k] = rng.choice(edges, k, replace=False)
        if r % 2:
            v[d // 2:] = v[:d - d // 2]  # every value twice
        src.append(np.full(d, (n - 1) // len(LENGTHS) * r))
        dst.append(v)
    src, dst = np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)
    p = rng.permutation(len(src))
    src, dst = np.ascontiguousarray(src[p]), np.ascontiguousarray(dst[p])
    g = gb.Graph.from_edges(n, src, dst, gb.DEDUP | (gb.WIDE_ROWS if wide else 0))
    o = orc.csr_build(n, src, dst, orc.DEDUP)
    row, col = g.csr()
    assert np.array_equal(row, o.row_offset)
    assert np.array_equal(col, o.col_idx)


def test_many_long_rows(gb, orc):
    """More rows than clusters are launched: bitmaps are left clear for the next row."""
    n, rows, d = 3000, 2900, 4200
    rng = np.random.default_rng(3)
    src = np.repeat(np.arange(rows), d).astype(np.int32)
    dst = rng.integers(0, n, rows * d).astype(np.int32)
    g = gb.Graph.from_edges(n, src, dst, gb.DEDUP)
    o = orc.csr_build(n, src, dst, orc.DEDUP)
    row, col = g.csr()
    assert np.array_equal(row, o.row_offset)
    assert np.array_equal(col, o.col_idx)
