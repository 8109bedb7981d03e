"""GPU parity of the label-correcting kernel over fixed-width rows where a
frontier is too wide for the CTAs' local ones: it goes from the global queue to
the next straight away, rows linked or not, and back to hops as it shrinks."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(gb, kind: str):
    rng = np.random.default_rng(7)
    if kind == "random 4-regular":
        n = 2_500_000
        v = np.arange(n)
        return n, np.concatenate([v, v]), np.concatenate([rng.permutation(n), rng.permutation(n)])
    if kind == "binary tree":
        n = 4_000_003
        return n, (np.arange(1, n) - 1) // 2, np.arange(1, n)
    n = 3_000_000  # a ring with shortcuts: 0.8 % of the rows linked
    v, m = np.arange(n), n // 5
    return n, np.concatenate([v, rng.integers(0, n, m)]), np.concatenate([(v + 1) % n, rng.integers(0, n, m)])


@pytest.mark.parametrize("kind,flags", [("random 4-regular", 0), ("random 4-regular", 16), ("binary tree", 0), ("ring", 0), ("ring", 16)])
def test_wide_frontiers(gb, orc, kind, flags):
    n, src, dst = _graph(gb, kind)
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    g = gb.Graph.from_edges(n, src, dst, gb.UNDIRECTED | flags)
    assert g.max_degree <= 16
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    for s0 in (0, n - 1):
        got, st = g.bfs(s0, stats=True)
        want = orc.bfs_queue(o, s0)
        assert np.array_equal(got, want)
        assert st.launches == 2 and st.levels == int(want.max()) + 1
        assert st.vertices_reached == int((want >= 0).sum())
        assert st.edges_in_component == orc.component_edges(o, want)
