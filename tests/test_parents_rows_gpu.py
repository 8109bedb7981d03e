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


@pytest.mark.parametrize("order", ["hub_first", "hub_first_wide", "unsorted", "star_chain"])
def test_parents_offered(gb, orc, order):
    """Large symmetric graphs with rows that do not ascend: some levels offer themselves."""
    if order == "star_chain":  # light, heavy and split rows offer, below a dense core
        n, src, dst = _star_chain(4)
        rng = np.random.default_rng(5)
        u = rng.integers(n - 20_000, n, (2, 4_800_000)).astype(np.int32)
        src, dst = np.concatenate([src, u[0]]), np.concatenate([dst, u[1]])
    else:
        n = 1 << 19
        src, dst = gb.gen_rmat(19, 16, seed=9)
    o = orc.csr_build(n, src, dst, orc.SYMMETRIZE | orc.DROP_SELF_LOOPS | orc.DEDUP)
    assert o.row_offset[-1] >= 1 << 23
    if order == "unsorted":
        g = gb.Graph.from_csr(o.row_offset.astype(np.int32), _rotated(o))
    else:
        g = gb.Graph.from_edges(n, src, dst, gb.UNDIRECTED | gb.HUB_FIRST | (gb.WIDE_ROWS if "wide" in order else 0))
    deg = np.diff(o.row_offset)
    light = np.flatnonzero(deg > 0)
    for s in (0, int(np.argmax(deg)), int(light[np.argmin(deg[light])])):
        lv, par = g.bfs_parents(s)
        want = orc.bfs_queue(o, s)
        assert np.array_equal(lv, want)
        assert np.array_equal(par, orc.min_parents(o, want))


def _rotated(o):
    """The columns with every row's first entry moved to its end."""
    col = o.col_idx.copy()
    row = o.row_offset
    some = np.flatnonzero(np.diff(row) > 1)
    first = col[row[some]].copy()
    nxt = np.arange(1, len(col) + 1)
    nxt[-1] = len(col) - 1
    out = col[nxt]
    out[row[some + 1] - 1] = first
    single = np.flatnonzero(np.diff(row) == 1)
    out[row[single]] = col[row[single]]
    return np.ascontiguousarray(out)
