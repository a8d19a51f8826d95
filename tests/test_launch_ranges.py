"""Which fields of a batch's launch class a launch covers (csrc/multi.cu), on
the host: every field that takes part is inside the range, and a step in which
none can take part costs no look at the fields."""
import shutil
import subprocess
from pathlib import Path

import pytest

PKG = Path(__file__).resolve().parents[1] / "parareal-cc-cfv-split-gpu_b200"
CUDA = Path("/usr/local/cuda/include")

PROGRAM = r"""
#include <chrono>
#include <cstdio>
#include <cstring>
#include <random>
#include "multi.h"
using namespace ccfv;

static SweepField field(int inst, int slice, int jmin, int jmax) {
  SweepField f;
  std::memset(&f, 0, sizeof(f));
  f.inst = inst;
  f.slice = slice;
  f.jmin = jmin;
  f.jmax = jmax;
  f.groups = 3;
  return f;
}

int main() {
  std::mt19937 rng(7);
  auto below = [&](int n) { return (int)(rng() % n); };
  long bad = 0;
  for (int trial = 0; trial < 400; ++trial) {
    SweepClass K;
    K.kind = below(4);
    const int inst = 1 + below(5);
    std::vector<int> nlo;
    for (int i = 0; i < inst; ++i) {
      // fused: the last x sweep in the last step only, the joined one before it
      const bool fused = below(2), slices = below(2);
      const int J = 1 + below(6), S = 1 + below(5);
      const int jmin = fused && K.kind == 2 ? J - 1 : 0;
      const int jmax = fused && K.kind == 0 ? 1 : fused && K.kind == 3 ? J - 1 : J;
      nlo.push_back(below(S + 1));
      if (jmax > 0)
        for (int s = 0; s < (slices ? S : 1); ++s) {
          SweepField f = field(i, slices ? s : -1, jmin, jmax);
          f.smax = S;
          K.h.push_back(f);
        }
    }
    finish_class(K);
    for (int j = 0; j < 8; ++j)
      for (int s = 0; s < 6; ++s) {
        int lo = -1, hi = -1, first = -1, last = -1;
        for (int i = 0; i < (int)K.h.size(); ++i)
          if (field_active(K.h[i], j, s, nlo.data())) {
            if (first < 0) first = i;
            last = i;
          }
        const bool any = active_fields(K, j, s, nlo.data(), &lo, &hi);
        if (any != (first >= 0)) ++bad;
        if (any && !(lo >= 0 && lo <= first && last < hi && hi <= (int)K.h.size())) ++bad;
        if (any && K.kind == 2 && (lo != first || hi != last + 1)) ++bad;
      }
  }
  // 100,000 slices of 1000 fused steps
  SweepClass K;
  K.kind = 2;
  for (int i = 0; i < 100000; ++i) K.h.push_back(field(i / 64, i % 64, 999, 1000));
  finish_class(K);
  std::vector<int> nlo(2000, 0);
  const auto t0 = std::chrono::steady_clock::now();
  int lo, hi, launches = 0;
  for (int j = 0; j < 1000; ++j) launches += active_fields(K, j, 0, nlo.data(), &lo, &hi);
  const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  std::printf("%ld %d %d %d %.6f\n", bad, launches, lo, hi, s);
  // a look at every field in every step is 10^8 of them
  return bad || launches != 1 || lo != 0 || hi != 100000 || s > 0.02;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not CUDA.exists(), reason="no host compiler")
def test_launches_cover_the_fields_that_take_part(tmp_path):
    src, exe = tmp_path / "ranges.cpp", tmp_path / "ranges"
    src.write_text(PROGRAM)
    lib = PKG / "lib"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(PKG / "csrc"), "-I", str(CUDA), "-o",
                    str(exe), str(src), str(lib / "libccfv.so"), f"-Wl,-rpath,{lib}"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
