"""GPU parity of BFS-tree parents on rows of every walk: up to 64 entries,
longer, and past 4096 (pieces of 2048), ascending, hub-first and unsorted."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _star_chain(seed: int):
    """Hubs of every row class in a chain, their leaves shared with random
    others, so that long rows sit at levels 1, 2 and 3."""
    rng = np.random.default_rng(seed)
    degrees = (63, 64, 65, 2048, 4095, 4096, 4097, 9001, 64)
    n = 30_000
    src, dst = [], []
    for h, d in enumerate(degrees):
        src.append(np.full(d, h))
        dst.append(rng.choice(np.arange(len(degrees), n), d, replace=False))
        if h:
            src.append([h - 1])
            dst.append([h])
    return n, np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)


@pytest.mark.parametrize("order", ["ascending", "hub_first", "unsorted", "wide", "directed"])
def test_parents_row_classes(gb, orc, order):
    n, src, dst = _star_chain(3)
    flags = 0 if order == "directed" else gb.UNDIRECTED
    extra = {"hub_first": gb.HUB_FIRST, "wide": gb.WIDE_ROWS}.get(order, 0)
    o = orc.csr_build(n, src, dst, flags)
    if order == "unsorted":
        rng = np.random.default_rng(1)
        row, col = o.row_offset, o.col_idx.copy()
        for v in range(n):
            rng.shuffle(col[row[v]:row[v + 1]])
        g = gb.Graph.from_csr(row, col)
    else:
        g = gb.Graph.from_edges(n, src, dst, flags | extra)
    for s in (0, 4, 8, int(dst[0]), int(dst[-1])):
        lv, par = g.bfs_parents(s)
        want = orc.bfs_queue(o, s)
        assert np.array_equal(lv, want)
        assert np.array_equal(par, orc.min_parents(o, want))
