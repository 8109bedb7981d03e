"""CPU: an optional allocation that is refused is not asked for by every call
(tests/cpp/retry_test.cpp over gpu_graphs_gb300/csrc/retry.h), and the two that
searches make go through that rule."""
from __future__ import annotations

import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "gpu_graphs_gb300" / "csrc"


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = tmp_path_factory.mktemp("retry") / "retry_test"
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", str(CSRC), str(ROOT / "tests" / "cpp" / "retry_test.cpp"),
                    "-o", str(exe)], check=True)
    return lambda calls, refused: tuple(int(x) for x in subprocess.run([str(exe), str(calls), str(refused)], check=True,
                                                                      capture_output=True, text=True).stdout.split())


def test_first_call_tries(run):
    assert run(5, 0) == (1, 0)


@pytest.mark.parametrize("refused", [1, 2, 3, 10, 100, 5000, 100_000])
def test_refusals_cost_few_tries_and_recovery_comes(run, refused):
    tries, at = run(10 * refused + 5000, refused)
    assert tries <= 2 + refused.bit_length() + refused // 1024
    assert refused <= at <= 2 * refused + 1025  # tried again within as many calls as were refused, and 1,024 at most


def test_searches_ask_through_the_rule():
    text = (CSRC / "api.cu").read_text()
    for build, rule in (("csr_build_quads(g->csr", "quad_retry.due()"),):
        for m in re.finditer(re.escape(build), text):
            assert rule in text[:m.start()][-250:]
    parents = text[text.index("int gbfs_bfs_parents("):text.index("int gbfs_bfs_many(")]
    assert "piece_retry.due()" in parents[:parents.index("ms_prepare(")]
