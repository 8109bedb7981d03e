"""GPU parity, and time, of passes that find each entry's row as they walk the
entries, over runs of empty rows between two entries."""
from __future__ import annotations

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAPS = (0, 1, 30, 31, 32, 33, 63, 64, 65, 1023, 1055, 1056, 1057, 2048, 32 * 1024, 33 * 1024 + 31, 33 * 1024 + 32,
        33 * 1024 + 33, 70_000, 1_100_000)


def _rows_after_gaps(first: int):
    """Row ids with each of GAPS empty rows between two of them."""
    rows = [first]
    for gap in GAPS + GAPS[::-1]:
        rows.append(rows[-1] + 1 + gap)
    return np.array(rows)


@pytest.mark.parametrize("first,last,per_row", [(0, 0, 1), (5, 0, 3), (40_000, 100_000, 1), (0, 1, 90)])
def test_gaps(gb, orc, first, last, per_row):
    rows = _rows_after_gaps(first)
    n = int(rows[-1]) + 1 + last
    rng = np.random.default_rng(per_row)
    src = np.repeat(rows, per_row)
    dst = rng.choice(rows, len(src))
    src, dst = np.append(src, rows[:-1]).astype(np.int32), np.append(dst, rows[1:]).astype(np.int32)
    for flags, oflags in ((0, 0), (gb.UNDIRECTED, orc.UNDIRECTED)):
        o = orc.csr_build(n, src, dst, oflags)
        for g in (gb.Graph.from_edges(n, src, dst, flags), gb.Graph.from_csr(o.row_offset, o.col_idx)):
            for s0 in (rows[0], rows[len(rows) // 2], rows[-1]):
                for direction in (gb.DIR_OPTIMIZING, gb.DIR_BOTTOMUP):
                    g.set_params(direction=direction)
                    assert np.array_equal(g.bfs(int(s0)), orc.bfs_queue(o, int(s0))), (flags, s0, direction)


def test_one_long_gap_does_not_hold_a_pass(gb):
    """The first search of a directed graph (its transpose is built then): 20 M rows
    between two entries cost little beside the same rows behind the last entry."""
    n, k = 20_000_000, 1000
    src = np.arange(k).repeat(8).astype(np.int32)
    dst = np.random.default_rng(1).integers(0, n, 8 * k).astype(np.int32)

    def first_search(rows):
        best = 1e9
        for _ in range(3):
            with gb.Graph.from_edges(n, rows, dst, 0) as g:
                out = np.empty(n, np.int32)
                a = time.perf_counter()
                g.bfs(0, out=out)
                best = min(best, time.perf_counter() - a)
        return best

    without = first_search(src)
    split = src.copy()
    split[4 * k:] += n - k
    assert first_search(split) < 3 * without
