"""GPU parity: the label-correcting kernel over fixed-width adjacency (rows
of more than four entries are linked) and its switch to the CSR kernel."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _caterpillar(n: int, every: int, degrees, seed: int):
    """A shuffled path in which every `every`-th vertex gets leaves up to one
    of `degrees`."""
    rng = np.random.default_rng(seed)
    src, dst, nxt = [np.arange(n - 1)], [np.arange(1, n)], n
    for k, v in enumerate(range(every, n - 1, every)):
        extra = degrees[k % len(degrees)] - 2
        src.append(np.full(extra, v))
        dst.append(np.arange(nxt, nxt + extra))
        nxt += extra
    perm = rng.permutation(nxt)
    src, dst = np.concatenate(src), np.concatenate(dst)
    return nxt, perm[src].astype(np.int32), perm[dst].astype(np.int32), perm


# (4,): no row linked; then one row in 30 linked, of 5 to 16 entries (one
# further entry in the node, and all thirteen); every fourth path vertex
# linked: past one row in 16, the CSR kernel
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("every,degrees", [(3, (4,)), (40, (5, 15, 16)), (4, (5, 6))])
def test_linked_rows(gb, orc, every, degrees, wide):
    n, src, dst, perm = _caterpillar(5000, every, degrees, every)
    g = gb.Graph.from_edges(n, src, dst, gb.UNDIRECTED | (gb.WIDE_ROWS if wide else 0))
    assert g.max_degree == max(degrees)
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    for s0 in (perm[0], perm[2500], perm[n - 1]):
        got, st = g.bfs(int(s0), stats=True)
        want = orc.bfs_queue(o, int(s0))
        assert np.array_equal(got, want)
        assert st.launches == 2 and st.levels == int(want.max()) + 1
        assert st.vertices_reached == int((want >= 0).sum())
        assert st.edges_in_component == orc.component_edges(o, want)
