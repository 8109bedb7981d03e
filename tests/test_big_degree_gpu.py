"""GPU: top-down steps over a small queue with one long row, whatever the row
length from which rows are split over the grid (big_degree)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(gb, rows: int, long_row: int):
    """The source, `rows` vertices behind it, and behind those 10 leaves each but
    `long_row` behind the first."""
    src, dst, at = [np.zeros(rows, int)], [np.arange(1, rows + 1)], rows + 1
    for v in range(1, rows + 1):
        k = long_row if v == 1 else 10
        src.append(np.full(k, v))
        dst.append(np.arange(at, at + k))
        at += k
    n = at + 140_000  # past the sizes that one cluster searches
    return n, np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)


@pytest.mark.parametrize("big_degree", [32, 256, 1023, 1024, 1025, 1 << 20])
@pytest.mark.parametrize("long_row", [1000, 1023, 1024, 1025, 9000])
def test_levels(gb, orc, big_degree, long_row):
    n, src, dst = _graph(gb, 700, long_row)
    g = gb.Graph.from_edges(n, src, dst)
    o = orc.csr_build(n, src, dst, orc.UNDIRECTED)
    for direction in (gb.DIR_OPTIMIZING, gb.DIR_TOPDOWN):
        g.set_params(direction=direction, big_degree=big_degree)
        for s0 in (0, 1, 700, n - 140_001):
            assert np.array_equal(g.bfs(s0), orc.bfs_queue(o, s0)), (direction, s0)


def test_long_row_is_not_one_warps(gb):
    torch = pytest.importorskip("torch")
    n, src, dst = _graph(gb, 2000, 60_000)
    g = gb.Graph.from_edges(n, src, dst)
    out = torch.empty(n, dtype=torch.int32, device="cuda")

    def ms(big_degree):
        g.set_params(direction=gb.DIR_TOPDOWN, big_degree=big_degree)
        return float(np.median([g.bfs(0, out=out, stats=True)[1].ms for _ in range(15)][3:]))

    assert ms(1 << 20) < 3 * ms(256)
