"""GPU parity of CSR builds large enough to go through buckets of rows, and of
inputs of that size that may not (one row with most of the entries)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(orc, n: int, src, dst, undirected: bool):
    if undirected:
        o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
        return o.row_offset, o.col_idx
    key = np.sort(src.astype(np.int64) * n + dst)
    row = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(src, minlength=n), out=row[1:])
    return row, (key % n).astype(np.int32)


@pytest.mark.parametrize("undirected", [True, False])
@pytest.mark.parametrize("kind,n,m", [
    ("uniform", 300_007, 10_600_001),      # the last bucket partly filled
    ("uniform", 1 << 22, 10_600_000),      # the most vertices a word holds
    ("uniform", (1 << 22) + 1, 10_600_000),  # one more: straight to the rows
    ("rmat", 1 << 19, 12 << 20),          # hubs: buckets of uneven size
    ("star", 200_000, 10_600_000),         # one bucket holds nearly all: straight to the rows
    ("local", 1_000_000, 10_600_000),     # edges in order of their ends: straight to the rows
    ("dense", 12_500, 10_600_000),         # few buckets
])
def test_large_builds(gb, orc, kind, n, m, undirected):
    if not undirected:
        m *= 2
    rng = np.random.default_rng(n)
    if kind == "rmat":
        src, dst = gb.gen_rmat(19, 24 if undirected else 48, seed=5)
    else:
        src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
        if kind == "local":
            src = np.arange(m) * n // m
            dst = np.minimum(src + rng.integers(0, 3, m), n - 1)
        if kind == "star":
            src[rng.random(m) < 0.9] = 77
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    g = gb.Graph.from_edges(n, src, dst, gb.UNDIRECTED if undirected else 0)
    row, col = g.csr()
    want_row, want_col = _csr(orc, n, src, dst, undirected)
    assert np.array_equal(row, want_row)
    assert np.array_equal(col, want_col)


def test_large_build_refuses_bad_ids(gb):
    src = np.zeros(22_000_000, np.int32)
    dst = np.arange(22_000_000, dtype=np.int32) % 300_000
    dst[-1] = 300_000
    with pytest.raises(gb.GbfsError):
        gb.Graph.from_edges(300_000, src, dst, 0)
