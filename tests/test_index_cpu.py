"""CPU: index arithmetic of the kernels at the end of the 32-bit range.

tests/cpp/index_test.cpp includes gpu_graphs_gb300/csrc/index.h (the walks the
kernels make) and runs them over ranges that end at 2^31 - 1, with traps on
signed overflow.
"""
from __future__ import annotations

import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "gpu_graphs_gb300" / "csrc"


def test_walks_at_the_end_of_the_index_range(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "index_test"
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-Wno-unknown-pragmas", "-ftrapv", "-I", str(CSRC),
                    str(ROOT / "tests" / "cpp" / "index_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_buckets_are_walked_by_the_checked_loop():
    """A build by buckets admits inputs whose last bucket ends at 2^31 - 1."""
    text = (CSRC / "csr_build.cu").read_text()
    body = text[text.index("k_bucket_rows(const BucketPlan"):text.index("struct BinLists")]
    assert body.count("walk_range<BK_BLOCK, BK_ILP>(s, e, t,") == 2
    assert "i0" not in body


# kernels whose rows may end at 2^31 - 1, and forms of their index arithmetic that
# leave the type there
PLAIN = [r"\(lo \+ hi\) *>> *1", r"\+= *(128|32 \* ILP)\b", r"\b(b|rb) \+ (MS_PIECE(?! - 1)|j \* )", r"\bi0 \+ t \* 32"]


@pytest.mark.parametrize("name", ["parents.cu", "msbfs.cu"])
def test_rows_are_walked_by_checked_arithmetic(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for pattern in PLAIN:
        assert not re.search(pattern, text), pattern


def test_bottom_up_probes_stay_in_range():
    text = re.sub(r"//[^\n]*", "", (CSRC / "bfs.cu").read_text())
    body = text[text.index("void probe_rows("):text.index("k_bfs(BfsArgs a)")]
    assert not re.search(r"\+= *(32|PROBE)\b|\bi[ab0]? *\+ *\(?(t|RT)\b[^;]*<|\bi0? < re\b", body)
    assert "+ skip < re" not in text and "+= two" not in text


def test_symmetry_check_halves_without_overflow():
    text = (CSRC / "csr_build.cu").read_text()
    body = text[text.index("bool row_has(const RT"):text.index("k_check_sorted(const RT")]
    assert "idx_mid(lo, hi)" in body and not re.search(PLAIN[0], body)
