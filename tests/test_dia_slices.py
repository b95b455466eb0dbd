"""Which slices count as diagonals: offsets whose product with the number of
right-hand sides leaves 32 bits do not (no GPU needed)."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpumatfun_gb300", "csrc")

# a band of 320 rows with couplings at +-40, found with a reach of 40 and of 39
PROGRAM = r"""
#include <cstdio>
#include "dia_slices.cuh"
struct Csr { std::vector<long long> ptr; std::vector<int> col; };
int main() {
  Csr A;
  A.ptr.push_back(0);
  for (int r = 0; r < 320; ++r) {
    for (int o : {-40, 0, 40})
      if (r + o >= 0 && r + o < 320) A.col.push_back(r + o);
    A.ptr.push_back((long long)A.col.size());
  }
  for (int diag_first = 0; diag_first < 2; ++diag_first)
    for (int reach : {40, 39}) {
      const gm::DiaSlices D = gm::find_dia(A, {0, 320}, {0, 10}, diag_first != 0, reach);
      std::printf("%d %d %lld %d\n", diag_first, reach, D.count, (int)D.len.size());
    }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_reach(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    # of ten slices 1 and 8 have rows with a neighbour outside; 0 and 9 have two
    # offsets, 2..7 three
    assert out[:4] == ["0 40 8 3", "0 39 0 0", "1 40 8 3", "1 39 0 0"]


def test_engine_passes_what_32_bits_hold():
    engine = open(os.path.join(CSRC, "engine.cu")).read()
    assert re.search(r"find_dia\(A, prow0, pslice0, diag_first, INT_MAX / e->R\)", engine)
