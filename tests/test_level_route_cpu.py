"""CPU: which batch outputs a kernel stores to (memory of the graph's own GPU) and
which are copied (another GPU's, which a kernel may not reach)."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "gpu_graphs_gb300" / "csrc"


def test_routes(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "level_route_test"
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC), str(ROOT / "tests" / "cpp" / "level_route_test.cpp"),
                    "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout.strip() == "ok"


def test_the_batch_takes_them():
    text = (CSRC / "batch.cu").read_text()
    body = text[text.index("int gbfs_bfs_batch("):text.index("int gbfs_bfs_batch_graphs(")]
    assert "output_route(levels_out[i], g->device)" in body
    assert "routes[i] == LevelRoute::KERNEL ? levels_out[i] : nullptr" in body
    assert "cudaMemcpyDeviceToDevice" in body[body.index("LevelRoute::COPY)\n            e ="):]
