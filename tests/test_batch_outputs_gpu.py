"""GPU: device outputs of a batch that one kernel cannot store to, or not in any
order: unaligned ones, and ones that overlap (the last member's levels stand)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(gb, orc, count):
    graphs = [(500 + 37 * i, *gb.gen_er(500 + 37 * i, 2000, i)) for i in range(count)]
    want = [orc.bfs_queue(orc.csr_build(n, s, d, orc.UNDIRECTED), 0) for n, s, d in graphs]
    return gb.GraphSet.from_edges(graphs), want


def _run(gb, gset, ptrs):
    src = np.zeros(len(ptrs), np.int32)
    arr = (C.c_void_p * len(ptrs))(*ptrs)
    assert gb.lib.gbfs_bfs_batch(gset._h, C.c_void_p(src.ctypes.data), C.cast(arr, C.c_void_p), None) == gb._lib.OK


def test_unaligned_outputs(gb, orc):
    torch = pytest.importorskip("torch")
    gset, want = _batch(gb, orc, 5)
    buf = [torch.zeros(4 * len(w) + 8, dtype=torch.uint8, device="cuda") for w in want]
    torch.cuda.synchronize()
    _run(gb, gset, [b.data_ptr() + i for i, b in enumerate(buf)])
    for i, (b, w) in enumerate(zip(buf, want)):
        assert np.array_equal(b.cpu().numpy()[i:i + 4 * len(w)].copy().view(np.int32), w), i


@pytest.mark.parametrize("order", [(0, 1, 2, 3), (3, 1, 0, 2)])
def test_overlapping_outputs(gb, orc, order):
    torch = pytest.importorskip("torch")
    gset, want = _batch(gb, orc, 4)
    n = max(map(len, want)) + 400
    buf = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    offset = [100 * k for k in order]
    for _ in range(3):
        buf.fill_(-7)
        torch.cuda.synchronize()
        _run(gb, gset, [buf.data_ptr() + 4 * o for o in offset])
        expect = np.full(n, -7, np.int32)
        for o, w in zip(offset, want):
            expect[o:o + len(w)] = w
        assert np.array_equal(buf.cpu().numpy(), expect)
    _run(gb, gset, [buf.data_ptr()] * 4)  # one buffer for all
    for w in want:
        expect[:len(w)] = w
    assert np.array_equal(buf.cpu().numpy(), expect)
