"""GPU parity of gbfs_bfs_batch outputs: device arrays, host arrays and both,
members of one vertex up to several copy blocks, at odd offsets."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["device", "mixed", "host"])
@pytest.mark.parametrize("sizes", [(1,), (4095, 1, 4096, 4097), (1,) * 300 + (9001, 3, 2, 50_000, 1)])
def test_batch_outputs(gb, orc, sizes, where):
    torch = pytest.importorskip("torch")
    members = []
    for i, n in enumerate(sizes):
        src, dst = gb.gen_er(n, 3 * n, i)
        members.append((n, src, dst))
    gs = gb.GraphSet.from_edges(members)
    roots = np.array([(7 * i) % n for i, n in enumerate(sizes)], np.int32)
    # one entry between the members' arrays on the device, so none is aligned
    pool = torch.full((sum(sizes) + len(sizes),), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ptrs, host, at = [], {}, 0
    for i, n in enumerate(sizes):
        if where == "device" or (where == "mixed" and i % 3):
            ptrs.append(pool.data_ptr() + 4 * (at + i))
        else:
            host[i] = np.full(n, -7, np.int32)
            ptrs.append(host[i].ctypes.data)
        at += n
    arr = (ctypes.c_void_p * len(ptrs))(*ptrs)
    for _ in range(2):
        gb.check(gb.lib.gbfs_bfs_batch(gs._h, roots.ctypes.data, arr, None), "gbfs_bfs_batch")
    got, at = pool.cpu().numpy(), 0
    for i, (n, src, dst) in enumerate(members):
        want = orc.bfs_queue(orc.csr_build(n, src, dst, orc.UNDIRECTED), int(roots[i]))
        part = host[i] if i in host else got[at + i:at + i + n]
        assert np.array_equal(part, want), i
        assert got[at + i + n] == -7  # the entry after it is untouched
        at += n
