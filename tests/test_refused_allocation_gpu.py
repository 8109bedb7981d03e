"""GPU: a call that the device has no memory for is refused, and the next one is not."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_after_a_refused_one(gb, orc):
    n = 900_000_000  # a 64-lane workspace takes 340 bytes a vertex: 306 GB
    src, dst = gb.gen_er(50_000, 200_000, 3)
    o = orc.csr_build(50_000, src, dst, orc.UNDIRECTED)
    out = np.empty((1, n), np.int32)
    with gb.Graph.from_edges(n, np.zeros(1, np.int32), np.ones(1, np.int32)) as large:
        for _ in range(2):
            with pytest.raises(gb.GbfsError) as e:
                large.bfs_multi([0], out=out)
            assert e.value.code == gb._lib.ERR_OOM
            with gb.Graph.from_edges(50_000, src, dst) as g:
                lv, par = g.bfs_parents(0)
                assert np.array_equal(lv, orc.bfs_queue(o, 0)) and (par >= 0).sum() == (lv > 0).sum()
                assert np.array_equal(g.bfs_multi([0, 7])[1], orc.bfs_queue(o, 7))
