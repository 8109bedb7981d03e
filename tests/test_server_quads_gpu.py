"""GPU: the fixed-width adjacency of small-degree graphs and a server's budget.
What the device holds for an admitted graph is in the budget, and no graph is
refused for the sake of another one's adjacency."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE = 400
N = SIDE * SIDE


class Grid:
    """The graph, its levels, and what a server counts for it."""

    def __init__(self, gb, orc):
        self.gb = gb
        self.src, self.dst = gb.gen_grid(SIDE, 0.1, 0.001, 8, 1)
        o = orc.csr_build(N, self.src, self.dst, orc.UNDIRECTED)
        self.levels = {s: orc.bfs_queue(o, s) for s in (0, N // 2, N - 1)}
        up = lambda b: (b + 255) & ~255
        self.quads = up(16 * N) + up(64 * int((np.diff(o.row_offset) > 4).sum())) + 256
        g = self.make()
        before = g.info()["device_bytes"]
        g.bfs(0)
        self.work = g.info()["device_bytes"] - before - self.quads  # of direct searches: in no server's budget
        assert self.work > 0
        with gb.Server(mem_budget_bytes=8 << 30, num_slots=2) as srv:
            srv.add_graph(self.make())
            st = srv.stats()
        self.slots, self.one = st["peak_bytes"] - st["resident_bytes"], st["resident_bytes"]

    def make(self):
        return self.gb.Graph.from_edges(N, self.src, self.dst)

    def held(self, g, searched: bool) -> int:
        return g.info()["device_bytes"] - (self.work if searched else 0)


@pytest.fixture(scope="module")
def grid(gb, orc):
    return Grid(gb, orc)


def _serve(srv, gid, grid):
    for s, want in grid.levels.items():
        assert np.array_equal(srv.wait(srv.submit(gid, s))[0], want)


@pytest.mark.parametrize("searched", [False, True])
def test_no_room_for_the_adjacency(gb, grid, searched):
    g = grid.make()
    plain = grid.held(g, False)
    if searched:
        assert np.array_equal(g.bfs(0), grid.levels[0])
        assert grid.held(g, True) == plain + grid.quads
    with gb.Server(mem_budget_bytes=grid.slots + grid.one - grid.quads // 2, num_slots=2) as srv:
        gid = srv.add_graph(g)
        resident = srv.stats()["resident_bytes"]
        # all that the device holds for the graph is counted
        assert grid.held(g, searched) <= resident <= grid.one - grid.quads // 2
        _serve(srv, gid, grid)
        for s, want in grid.levels.items():
            assert np.array_equal(g.bfs(s), want)
        assert grid.held(g, True) <= resident  # direct searches do not build it either
        srv.remove_graph(gid)
        assert np.array_equal(g.bfs(0), grid.levels[0])
        assert grid.held(g, True) > plain + grid.quads - 1  # admitted nowhere: built


def test_room_for_a_built_adjacency(gb, grid):
    g = grid.make()
    g.bfs(0)
    with gb.Server(mem_budget_bytes=grid.slots + grid.one, num_slots=2) as srv:
        gid = srv.add_graph(g)
        assert grid.held(g, True) <= srv.stats()["resident_bytes"] <= grid.one
        _serve(srv, gid, grid)


def test_a_later_graph_takes_the_adjacencies_room(gb, grid):
    graphs = [grid.make() for _ in range(3)]
    budget = grid.slots + 3 * grid.one - 2 * grid.quads  # three graphs with one adjacency among them
    with gb.Server(mem_budget_bytes=budget, num_slots=2) as srv:
        ids = [srv.add_graph(graphs[0])]
        with_quads = grid.held(graphs[0], False)
        sources = list(grid.levels) * 20
        tickets = [srv.submit(ids[0], s) for s in sources]
        ids += [srv.add_graph(g) for g in graphs[1:]]
        held = [grid.held(g, False) for g in graphs]
        assert min(held) == with_quads - grid.quads
        assert sum(held) <= srv.stats()["resident_bytes"] <= budget - grid.slots
        for t, s in zip(tickets, sources):
            assert np.array_equal(srv.wait(t)[0], grid.levels[s])
        for gid in ids:
            _serve(srv, gid, grid)
        assert srv.stats()["rejected"] == 0
        with pytest.raises(gb.GbfsError) as e:
            srv.add_graph(grid.make())
        assert e.value.code == gb._lib.ERR_BUDGET
        for gid in ids:
            srv.remove_graph(gid)
        assert srv.stats()["resident_bytes"] == 0


def test_an_adjacency_that_another_server_uses(gb, grid):
    """It stays in that one's budget; the other server gives up its use, not the graph."""
    shared, other = grid.make(), grid.make()
    plain = grid.held(shared, False)
    tight_budget = grid.slots + 2 * grid.one - grid.quads - grid.quads // 2  # one adjacency of two graphs too much
    with gb.Server(mem_budget_bytes=8 << 30, num_slots=2) as roomy, gb.Server(mem_budget_bytes=tight_budget, num_slots=2) as tight:
        a, b = roomy.add_graph(shared), tight.add_graph(shared)
        c = tight.add_graph(other)
        assert tight.stats()["resident_bytes"] <= tight_budget - grid.slots
        assert grid.held(shared, False) == plain + grid.quads <= roomy.stats()["resident_bytes"]
        for srv, gid in ((roomy, a), (tight, b), (tight, c)):
            _serve(srv, gid, grid)
        roomy.remove_graph(a)  # nobody's any more
        assert grid.held(shared, False) == plain
        _serve(tight, b, grid)
        _serve(tight, c, grid)
