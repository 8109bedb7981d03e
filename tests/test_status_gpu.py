"""GPU: a search that some CTA has left early is reported, whatever the others
wrote, and leaves nothing behind for the next one."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(gb, kind: str):
    if kind == "power law":  # the grid kernel, to its end
        n = 1 << 18
        src, dst = gb.gen_rmat(18, 8, seed=3)
    else:  # parked for the label-correcting kernel (on its fixed-width rows, or the rows themselves)
        n = 300 * 300
        src, dst = gb.gen_grid(300, 0.0, 0.0, 1, 1)
        if kind == "mesh":  # diagonals: rows of six entries
            v = np.arange(n).reshape(300, 300)
            src = np.concatenate([src, v[:-1, :-1].ravel()]).astype(np.int32)
            dst = np.concatenate([dst, v[1:, 1:].ravel()]).astype(np.int32)
    return n, src, dst


@pytest.mark.parametrize("kind,per_level", [("power law", 0), ("power law", 1), ("power law", 2), ("grid", 0), ("mesh", 0)])
def test_marked_search_is_reported_and_cleared(gb, orc, kind, per_level):
    n, src, dst = _graph(gb, kind)
    g = gb.Graph.from_edges(n, src, dst)
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    g.set_params(per_level_launch=per_level)
    s0 = int(src[0])
    want = orc.bfs_queue(o, s0)
    calls = [lambda: g.bfs(s0), lambda: g.bfs_multiroot([s0]), lambda: g.bfs_many([s0, s0, s0])[0][2]]
    for call in calls:
        assert np.array_equal(call(), want)
        assert gb.lib.gbfs_selftest_mark_timeout(g.handle) == gb._lib.OK
        with pytest.raises(gb.GbfsError) as e:
            call()
        assert e.value.code == gb._lib.ERR_TIMEOUT
        for _ in range(2):
            assert np.array_equal(call(), want)


def test_mark_needs_a_searched_graph(gb):
    g = gb.Graph.from_edges(3, [0, 1], [1, 2])
    assert gb.lib.gbfs_selftest_mark_timeout(g.handle) == gb._lib.ERR_INVALID_ARG
    assert gb.lib.gbfs_selftest_mark_timeout(None) == gb._lib.ERR_INVALID_ARG
