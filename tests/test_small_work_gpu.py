"""GPU: searches on one cluster take a workspace without queues, which searches
of the same graph that need them add."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n", [1000, 30_000, 131_072])
def test_workspace_grows_with_need(gb, orc, n, wide):
    src, dst = gb.gen_er(n, 3 * n, 3)
    src, dst = np.append(src, np.zeros(30, np.int32)), np.append(dst, np.arange(1, 31, dtype=np.int32))  # a row past 16
    flags = gb.UNDIRECTED | (gb.WIDE_ROWS if wide else 0)
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    want = orc.bfs_queue(o, 0)

    def fresh():
        g = gb.Graph.from_edges(n, src, dst, flags)
        return g, g.info()["device_bytes"]

    def grown(g, before):
        return g.info()["device_bytes"] - before

    g, before = fresh()
    assert np.array_equal(g.bfs(0), want)
    small = grown(g, before)
    assert small < 9 * n + 16384 * 40 + 4096  # levels, staged roots, the control block
    g.set_params(direction=gb.DIR_BOTTOMUP)
    assert np.array_equal(g.bfs(0), want)
    assert grown(g, before) > small + 24 * n
    for direction in (gb.DIR_OPTIMIZING, gb.DIR_TOPDOWN, gb.DIR_BOTTOMUP):
        for per_level in ((0,) if wide else (0, 1, 2)):
            g.set_params(direction=direction, per_level_launch=per_level)
            assert np.array_equal(g.bfs(0), want)
            assert np.array_equal(g.bfs_multiroot([0]), want)
            assert np.array_equal(g.bfs_many([0, 0])[0][1], want)
    # every other call first, on a graph with a small workspace or none
    for searched in (False, True):
        for call in (lambda g: g.bfs_parents(0)[0], lambda g: g.bfs_many([0, 0, 0])[0][2], lambda g: g.bfs_multiroot([0]),
                     lambda g: (g.set_params(per_level_launch=0 if wide else 2), g.bfs(0))[1]):
            g, _ = fresh()
            if searched:
                g.bfs(n - 1)
            assert np.array_equal(call(g), want)
            assert np.array_equal(g.bfs(0), want)


def test_parents_with_host_and_device_outputs(gb, orc):
    torch = pytest.importorskip("torch")
    n = 20_000
    src, dst = gb.gen_er(n, 5 * n, 4)
    src, dst = np.append(src, np.zeros(30, np.int32)), np.append(dst, np.arange(1, 31, dtype=np.int32))
    for flags in (gb.UNDIRECTED, 0):
        g = gb.Graph.from_edges(n, src, dst, flags)
        lv, par = g.bfs_parents(0)
        tl, tp = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
        g.bfs_parents(0, levels=tl, parents=tp)
        assert np.array_equal(tl.cpu().numpy(), lv) and np.array_equal(tp.cpu().numpy(), par)
        row, col = g.csr()
        u = np.repeat(np.arange(n), np.diff(row))
        ok = (lv[u] >= 0) & (lv[col] == lv[u] + 1)
        best = np.full(n, np.iinfo(np.int32).max)
        np.minimum.at(best, col[ok], u[ok])
        assert np.array_equal(par, np.where(lv > 0, best, -1))
