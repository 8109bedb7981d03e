"""CPU: synchronisation that the CUDA programming model asks for and that a run
cannot show to be missing, read from the kernels' source."""
from __future__ import annotations

import re

import pytest

from conftest import ROOT

CSRC = ROOT / "gpu_graphs_gb300" / "csrc"
BARRIER = re.compile(r"\bcluster_barrier\s*\(|barrier\.cluster\.(arrive|wait)")
REMOTE = re.compile(r"\bremote_(load|store)_\w+\s*\(|\b(ld|st|atom|red)\.shared::cluster")


def kernels() -> dict[str, str]:
    """Every __global__ function's body, without comments."""
    out = {}
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read_text(), flags=re.S)
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth, i = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
                if depth == 0:
                    break
            out[m.group(1)] = text[start:i]
    return out


REMOTE_KERNELS = sorted(k for k, body in kernels().items() if REMOTE.search(body))


def test_kernels_are_found():
    assert {"k_bfs", "k_bfs_small", "k_long_rows"} <= set(kernels())
    assert {"k_bfs_small", "k_long_rows"} <= set(REMOTE_KERNELS)


@pytest.mark.parametrize("name", REMOTE_KERNELS)
def test_remote_shared_memory_lies_between_cluster_barriers(name):
    """A CTA's shared memory may be accessed from another one only after it has
    started and before it ends."""
    body = kernels()[name]
    barriers = [m.start() for m in BARRIER.finditer(body)]
    remote = [m.start() for m in REMOTE.finditer(body)]
    assert barriers and barriers[0] < remote[0], "no cluster barrier before the first remote access"
    assert barriers[-1] > remote[-1], "no cluster barrier after the last remote access"


def test_small_search_reads_a_word_of_new_vertices_before_it_is_cleared():
    """All lanes of a warp read the word that one of them clears."""
    body = kernels()["k_bfs_small"]
    read = body.index("= sh.fresh[v >> 5]")
    clear = body.index("sh.fresh[v >> 5] = 0")
    assert read < clear and "__syncwarp()" in body[read:clear]


def test_builds_that_fail_wait_for_their_copies():
    """A pinned slot goes back to all users of the pool at the end of its scope: a
    function that copies into one synchronises before it returns an error."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "csr_build.cu").read_text())
    functions = re.split(r"\n(?=(?:template [^\n]*\n)?(?:int|struct|cudaError_t|void) \w)", text)
    holders = [f for f in functions if re.search(r"\bPinned<\w+> \w+;|\bRowSorter<RT> \w+;", f) and "done:" in f]
    assert len(holders) == 5
    for f in holders:
        assert "if (rc) cudaStreamSynchronize(st);" in f[f.rindex("done:"):], f[:200]
