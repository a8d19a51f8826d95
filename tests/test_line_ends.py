"""The per-edge formulas of the line ends (csrc/line_ends.cuh) compiled for the
host: a foot whose cells are not staged is reported and reads nothing, every
other foot reads staged cells only and gives what the whole line gives."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "parareal-cc-cfv-split-gpu_b200" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <initializer_list>
#define __device__
#define __forceinline__ inline
#include "line_ends.cuh"
using namespace ccfv;

const int L = 40;
double cell[L + 4];  // C_{-2} .. C_{L+1}
struct Line {        // positions [b0, b1) are staged
  int b0, b1;
  mutable long outside = 0;
  double operator()(int p) const {
    if (p < b0 || p >= b1 || p < -2 || p > L + 1) { ++outside; return 0; }
    return cell[p + 2];
  }
  bool near(int k) const { return k - 3 >= b0 && k + 3 < b1; }
};

template <bool REMAPPED>
long run(int b0, int b1, long *rejected) {
  long bad = 0;
  for (int k = -1; k <= L; ++k)
    for (int mark : {k, FOOT_BELOW, FOOT_ON_END, FOOT_ABOVE + L - 1, FOOT_ABOVE + L}) {
      // a mark of a foot inside the line, or of one clamped to its ends
      const bool inner = k >= 2 && k <= L - 4;
      if (inner ? mark != k : (k < 0 || k >= L) && mark == k) continue;
      auto end_cell = [&] { return FootCell{k < L / 2 ? 0 : L - 1, 0.25}; };
      Line part{b0, b1}, whole{-100, L + 100};
      double phi = k, d = 0.375, phw = k, dw = 0.375;
      const bool ok = foot_inputs<REMAPPED>(part, L, 1.0, mark, true, end_cell, phi, d);
      foot_inputs<REMAPPED>(whole, L, 1.0, mark, true, end_cell, phw, dw);
      bad += part.outside;
      if (ok != part.near(k)) ++bad;
      if (ok ? phi != phw || d != dw : phi != 0 || d != 0) ++bad;
      *rejected += !ok;
    }
  double phi = NO_CELL, d = 0.375;
  Line none{7, 7};
  if (!foot_inputs<REMAPPED>(none, L, 1.0, FOOT_BELOW, true, [] { return FootCell{0, 0.0}; }, phi, d) ||
      phi != 0 || d != 0 || none.outside)
    ++bad;
  return bad;
}

int main() {
  for (int i = 0; i < L + 4; ++i) cell[i] = std::sin(0.7 * i) + 2;
  long bad = 0, rejected = 0;
  for (int b0 : {-6, -2, 0, 5, 21, 30})
    for (int b1 : {12, 20, L, L + 2, L + 6}) {
      if (b1 <= b0) continue;
      bad += run<false>(b0, b1, &rejected) + run<true>(b0, b1, &rejected);
    }
  std::printf("%ld %ld\n", bad, rejected);
  return bad != 0 || rejected == 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_a_foot_outside_the_staged_cells_reads_nothing(tmp_path):
    src = tmp_path / "line_ends.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "line_ends"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-o", str(exe), str(src)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
