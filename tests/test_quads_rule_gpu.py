"""GPU: which graphs get the fixed-width adjacency (their first search adds at
least 16 bytes a vertex for it), with levels as the oracle's either way."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WORK = 5 * 4 + 2 * 8 + 1  # bytes a vertex of a search's workspace: five int arrays, two of row bounds, bitmaps


def _ring(n: int, share: float, seed: int = 1):
    """A ring in which `share` of the vertices have three leaves less or more: rows of five."""
    rng = np.random.default_rng(seed)
    k = int(share * n)
    v = np.arange(n)
    hubs = rng.choice(n, k, replace=False)
    return n + 3 * k, np.concatenate([v, np.repeat(hubs, 3)]), np.concatenate([(v + 1) % n, np.arange(n, n + 3 * k)])


def _graph(gb, kind: str):
    if kind == "grid":
        return 200 * 200, *gb.gen_grid(200, 0.1, 0.001, 8, 1)
    if kind == "sparse random":  # 13 % of the vertices without edges, 5 % of the rows longer than four
        return 200_000, *gb.gen_er(200_000, 200_000, 3)
    if kind == "sparser random":  # 30 % and 0.8 %
        return 200_000, *gb.gen_er(200_000, 120_000, 3)
    share, n = {"3 %": (0.032, 50_000), "4 %": (0.038, 50_000), "1.4 %": (0.0145, 1_200_000), "2 %": (0.021, 1_200_000)}[kind]
    return _ring(n, share)


@pytest.mark.parametrize("kind,quads", [("grid", True), ("sparse random", False), ("sparser random", False), ("3 %", True),
                                        ("4 %", False), ("1.4 %", True), ("2 %", False)])
def test_which_graphs_get_quads(gb, orc, kind, quads):
    n, src, dst = _graph(gb, kind)
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    g = gb.Graph.from_edges(n, src, dst)
    before = g.info()["device_bytes"]
    got = g.bfs(int(src[0]))
    added = g.info()["device_bytes"] - before - WORK * n - 16384 * 40 - 8192
    assert (added > 0) == quads, (added, added / n)
    assert np.array_equal(got, orc.bfs_queue(orc.csr_build(n, src, dst, orc.UNDIRECTED), int(src[0])))
