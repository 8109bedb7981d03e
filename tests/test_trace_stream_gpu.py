"""GPU: reading a search's trace does not wait for work on the default stream."""
from __future__ import annotations

import time

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multi", [False, True])
def test_trace_beside_a_busy_default_stream(gb, multi):
    torch = pytest.importorskip("torch")
    src, dst = gb.gen_rmat(14, 8, seed=1)
    g = gb.Graph.from_edges(1 << 14, src, dst)
    if multi:
        g.bfs_multi([0, 1])
    else:
        g.bfs(0)
    want = g.last_trace()
    torch.cuda.synchronize()
    torch.cuda._sleep(2_000_000_000)  # about a second
    a = time.perf_counter()
    got = g.last_trace()
    took = time.perf_counter() - a
    waited = time.perf_counter()
    torch.cuda.synchronize()
    assert time.perf_counter() - waited > 0.2  # the stream was busy all along
    assert got == want and took < 0.2
