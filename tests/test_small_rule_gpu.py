"""GPU: a small graph of which one part holds most of the entries, or one row,
is not searched by one cluster, where the CTA that owns it would keep the others
waiting: it takes about as long as the same graph beside enough isolated vertices
for the grid kernel.  Levels are the oracle's either way."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _edges(gb, kind: str):
    rng = np.random.default_rng(1)
    if kind.startswith("clique"):  # of the first c vertices, the others sparse
        c, n = {"clique 1000": (1000, 130_000), "clique 2000": (2000, 20_000)}[kind]
        i, j = np.triu_indices(c, 1)
        return n, np.append(i, rng.integers(0, n, 2 * n)), np.append(j, rng.integers(0, n, 2 * n))
    if kind == "dense":
        return 2000, *gb.gen_er(2000, 1_000_000, 3)
    if kind == "star":
        return 130_000, np.zeros(129_999, int), np.arange(1, 130_000)
    hubs = rng.integers(0, 4, 4 * 130_000)  # "hubs": the first four
    return 130_000, hubs, rng.integers(0, 130_000, 4 * 130_000)


def _ms(gb, g, s0, direction):
    torch = pytest.importorskip("torch")
    out = torch.empty(g.n, dtype=torch.int32, device="cuda")
    g.set_params(direction=direction)
    return float(np.median([g.bfs(s0, out=out, stats=True)[1].ms for _ in range(15)][3:]))


@pytest.mark.parametrize("kind", ["clique 1000", "clique 2000", "dense", "star", "hubs"])
@pytest.mark.parametrize("direction", [0, 1])
def test_one_part_with_most_entries(gb, orc, kind, direction):
    n, src, dst = _edges(gb, kind)
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    g = gb.Graph.from_edges(n, src, dst)
    big = gb.Graph.from_edges(140_000, src, dst)
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    for s0 in (0, n - 1):
        g.set_params(direction=direction)
        assert np.array_equal(g.bfs(s0), orc.bfs_queue(o, s0))
    assert _ms(gb, g, 0, direction) < 1.5 * _ms(gb, big, 0, direction)


@pytest.mark.parametrize("leaves", [510, 511, 512, 513, 16382, 16383, 16384, 16385, 33_000])
def test_levels_around_the_line(gb, orc, leaves):
    """Rows on both sides of the longest that one cluster takes, and parts on both
    sides of the most costly: several stars in one part."""
    for stars in (1, 2, 5):
        n = min(131_072, stars * leaves + 40)
        src, dst = [np.arange(39)], [np.arange(1, 40)]
        for k in range(stars):
            src.append(np.full(leaves, 7 * k))
            dst.append((40 + (k * leaves + np.arange(leaves)) % (n - 40)))
        src, dst = np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)
        g = gb.Graph.from_edges(n, src, dst)
        o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
        for direction in (0, 1):
            g.set_params(direction=direction)
            for s0 in (0, 39, n - 1):
                assert np.array_equal(g.bfs(s0), orc.bfs_queue(o, s0)), (stars, direction, s0)
