"""The gains of a butterfly and its inverse (round_trip in ws_codelets.cuh, from
gen_codelets.py's exact arithmetic on the rounded constants) against the
codelets run in single precision on random numbers: 1 + gain on each output of
inverse-then-forward and on each input of forward-then-inverse.

A sample's rounding is about 1e-7 of the mean square; over 40000 samples its
mean is 5e-10, and 4e-9 leaves room for eight times that.  The gains are up to
5e-8."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "wavesim_b200", "csrc")
CUDA_INC = "/usr/local/cuda/include"


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INC), reason="needs g++ and CUDA headers")
def test_gains_of_the_codelets(tmp_path):
    src = tmp_path / "gain.cpp"
    src.write_text(r"""#include <math.h>
#include <cstdio>
#include <random>
#include <cuda_runtime.h>
#include "ws_codelets.cuh"
template <int R, bool FIRST> void measure(int side) {
  std::mt19937 rng(7);
  std::normal_distribution<float> normal;
  double num[R] = {}, den[R] = {};
  for (int s = 0; s < 40000; ++s) {
    float2 x[R], v[R];
    for (int i = 0; i < R; ++i) x[i] = v[i] = make_float2(normal(rng), normal(rng));
    ws::Dft<R, FIRST>::run(v);
    ws::Dft<R, !FIRST>::run(v);
    for (int i = 0; i < R; ++i) {
      num[i] += (double)v[i].x * x[i].x + (double)v[i].y * x[i].y;
      den[i] += (double)x[i].x * x[i].x + (double)x[i].y * x[i].y;
    }
  }
  for (int i = 0; i < R; ++i)
    std::printf("%d %d %d %.9e %.9e\n", side, R, i, num[i] / den[i] / R - 1.0, ws::round_trip(side, R, i));
}
template <int R> void all() {
  if constexpr (R > 1) {
    measure<R, true>(0);
    measure<R, false>(1);
    all<R - 1>();
  }
}
int main() { all<16>(); }
""")
    exe = tmp_path / "gain"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, "-I", CUDA_INC, str(src), "-o", str(exe)], check=True)
    rows = np.loadtxt(subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.splitlines())
    assert len(rows) == 2 * sum(range(2, 17))
    assert np.abs(rows[:, 4]).max() > 3e-8
    assert np.abs(rows[:, 3] - rows[:, 4]).max() < 4e-9
