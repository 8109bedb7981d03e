"""GPU parity of the one-cluster search: vertex counts at the edges of its CTA
and cluster sizes, rows at its long-row edge, long searches, several roots."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(g, o, orc, sources):
    for s0 in sources:
        got, st = g.bfs(int(s0), stats=True)
        want = orc.bfs_queue(o, int(s0))
        assert np.array_equal(got, want), int(s0)
        assert st.launches == 1 and st.levels == int(want.max()) + 1
        assert st.vertices_reached == int((want >= 0).sum())
        assert st.edges_in_component == orc.component_edges(o, want)
        rows = [r for r in g.last_trace() if r["level"] >= 0]
        assert [r["level"] for r in rows] == list(range(st.levels))
        assert [r["frontier"] for r in rows] == np.bincount(want[want >= 0]).tolist()


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n", [31, 1023, 1024, 1025, 2049, 16384, 16385, 32769, 65536, 65537, 131071, 131072, 131073])
def test_vertex_counts(gb, orc, n, wide):
    src, dst = gb.gen_er(n, 5 * n, n)
    # a hub, so that the graph is not one of small degree; the last vertex too
    src, dst = np.append(src, np.zeros(30, np.int32)), np.append(dst, np.arange(n - 30, n, dtype=np.int32))
    g = gb.Graph.from_edges(n, src, dst, gb.UNDIRECTED | (gb.WIDE_ROWS if wide else 0))
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    for direction in (gb.DIR_OPTIMIZING, gb.DIR_TOPDOWN):
        g.set_params(direction=direction)
        _check(g, o, orc, (0, n // 2, n - 1))


def test_long_rows_and_long_searches(gb, orc):
    """Stars of 510 to 3000 leaves strung on a path of 700: levels past the
    trace rows held on chip, rows on both sides of the long-row edge."""
    n, src, dst = 700, [np.arange(699)], [np.arange(1, 700)]
    for k, leaves in enumerate((508, 509, 510, 511, 3000, 17)):
        src.append(np.full(leaves, 100 * k + 3))
        dst.append(np.arange(n, n + leaves))
        n += leaves
    src, dst = np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    _check(gb.Graph.from_edges(n, src, dst, gb.UNDIRECTED), o, orc, (0, 303, 699, n - 1))
    od = orc.csr_build(n, src, dst, 0)  # as stored: leaves are sinks
    _check(gb.Graph.from_edges(n, src, dst, 0), od, orc, (0, 403, n - 1))


def test_roots_and_back_to_back(gb, orc):
    n = 20_000
    src, dst = gb.gen_er(n, 6 * n, 9)
    src, dst = np.append(src, np.zeros(30, np.int32)), np.append(dst, np.arange(30, dtype=np.int32))
    g = gb.Graph.from_edges(n, src, dst)
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    roots = [5, n - 1, 5, 1024, 1023, 16384]
    got, st = g.bfs_multiroot(roots, stats=True)
    each = np.stack([orc.bfs_queue(o, r) for r in roots])
    want = np.where(each < 0, 1 << 30, each).min(0)
    assert np.array_equal(got, np.where(want == 1 << 30, -1, want))
    assert st.vertices_reached == int((want < 1 << 30).sum())
    outs, sts = g.bfs_many(roots)
    assert np.array_equal(outs, each) and all(s.launches == 1 for s in sts)
