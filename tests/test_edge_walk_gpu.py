"""GPU parity where the build walks entries in chunks of 1024 over rows of any
length: symmetry and order of a given CSR, and the transpose of a directed one."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(kind: str, seed: int):
    rng = np.random.default_rng(seed)
    if kind == "runs_of_empty_rows":  # 1000 empty rows between any two others
        a = rng.integers(0, 60, 900) * 1001
        return 60 * 1001, a, rng.permutation(a)
    if kind == "hub":  # one row over many chunks, then rows of one entry
        n = 9000
        return n, np.concatenate([np.zeros(n - 1, int), np.arange(1, n - 1)]), np.concatenate([np.arange(1, n), np.arange(2, n)])
    if kind == "last_row":  # every entry in the last row
        return 5000, np.full(4999, 4999), np.arange(4999)
    return 1, np.zeros(0, int), np.zeros(0, int)  # no entries


@pytest.mark.parametrize("kind", ["runs_of_empty_rows", "hub", "last_row", "empty"])
@pytest.mark.parametrize("shuffled", [False, True])
def test_given_csr(gb, orc, kind, shuffled):
    n, src, dst = _graph(kind, 3)
    for flags in (orc.UNDIRECTED, 0):
        o = orc.csr_build(n, src.astype(np.int32), dst.astype(np.int32), flags)
        row, col = o.row_offset, o.col_idx.copy()
        if shuffled:
            rng = np.random.default_rng(1)
            for v in np.flatnonzero(np.diff(row) > 1):
                rng.shuffle(col[row[v]:row[v + 1]])
        for drop in (False, True):  # the last entry of a symmetric graph left out
            if drop and (flags == 0 or len(col) == 0):
                continue
            if drop:
                row = np.minimum(row, len(col) - 1)
                col = col[:-1]
            g = gb.Graph.from_csr(row, col)
            c = orc.CSR(n, row, col)
            for s0 in (0, n - 1, n // 2):
                for direction in (gb.DIR_OPTIMIZING, gb.DIR_BOTTOMUP):
                    g.set_params(direction=direction)
                    assert np.array_equal(g.bfs(s0), orc.bfs_queue(c, s0)), (flags, drop, s0, direction)
