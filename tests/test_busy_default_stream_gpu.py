"""GPU: the first search of a graph is ordered after the clearing of its control
block whatever else is queued on the default stream."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(gb, kind: str):
    if kind == "power law":
        return 1 << 18, *gb.gen_rmat(18, 8, seed=3)
    if kind == "grid":
        return 300 * 300, *gb.gen_grid(300, 0.1, 0.001, 8, 1)
    return 20_000, *gb.gen_er(20_000, 100_000, 1)  # one cluster


@pytest.mark.parametrize("kind", ["power law", "grid", "small"])
def test_first_search(gb, orc, kind):
    torch = pytest.importorskip("torch")
    n, src, dst = _graph(gb, kind)
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    s0 = int(src[0])
    want = orc.bfs_queue(o, s0)
    calls = {"bfs": lambda g: g.bfs(s0), "many": lambda g: g.bfs_many([s0, s0])[0][1], "multiroot": lambda g: g.bfs_multiroot([s0]),
             "parents": lambda g: g.bfs_parents(s0)[0], "multi": lambda g: g.bfs_multi([s0, 0])[0]}
    for call in calls.values():  # kernels loaded
        g = gb.Graph.from_edges(n, src, dst)
        call(g)
        g.close()
    torch.zeros(1, device="cuda")
    for name, call in calls.items():
        g = gb.Graph.from_edges(n, src, dst)
        torch.cuda.synchronize()
        torch.cuda._sleep(1_000_000_000)  # half a second
        got = call(g)
        torch.cuda.synchronize()
        assert np.array_equal(got, want), name
        assert np.array_equal(call(g), want), name


def test_first_query_of_a_server(gb, orc):
    torch = pytest.importorskip("torch")
    n, src, dst = _graph(gb, "power law")
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    g = gb.Graph.from_edges(n, src, dst)
    torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    torch.cuda._sleep(1_000_000_000)
    with gb.Server(mem_budget_bytes=8 << 30, num_slots=2) as srv:
        gid = srv.add_graph(g)
        tickets = [srv.submit(gid, int(s)) for s in src[:8]]
        for t, s in zip(tickets, src[:8]):
            assert np.array_equal(srv.wait(t)[0], orc.bfs_queue(o, int(s)))
    torch.cuda.synchronize()
