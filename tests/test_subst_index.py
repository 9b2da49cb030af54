"""The substitutions (chol_subst.cuh) load a block's columns without a predicate and select the
values afterwards, so the addresses themselves have to stay inside the packed factor and the
kPanel elements behind it that every caller owns.  Walked here on the CPU, from the header the
kernels take them from, for every width of a problem the batched factorisation holds."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "s-pgo_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "subst_index.h"
using namespace spgo;
int main() {
  for (int P = 6; P <= 300; P += 6) {
    const int npk = P * (P + 1) / 2;
    auto cb = [&](int j) { return j * P - j * (j + 1) / 2; };
    for (int kb = 0; kb < P; kb += kPanel) {
      const int w = P - kb < kPanel ? P - kb : kPanel;
      for (int c0 = 0; c0 <= kPanel / 2; c0 += kPanel / 2)
        for (int i = 0; i < kPanel; ++i) {
          int at = cb(kb) + kb + i + subst_fwd_first(P, kb, c0);
          for (int c = c0; c < kPanel; ++c) {
            if (at < 0 || at >= npk + kPanel) return printf("P %d block %d row %d column %d: element %d of %d\n", P, kb, i, c, at, npk), 1;
            if (c <= i && i < w && at != cb(kb + c) + kb + i) return printf("P %d block %d row %d column %d: not its own element\n", P, kb, i, c), 1;
            at += subst_fwd_step(P, kb, c);
          }
        }
    }
  }
  return 0;
}
"""


def test_unconditional_loads_stay_in_the_factor(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
