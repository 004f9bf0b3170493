"""The bf16 digits of the split operands (oa_planes.cuh), compiled for the host:
as close to the value as digits taken from FP64 remainders.  No GPU."""
import os
import subprocess

import pytest

from openatom_b200 import build

SRC = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "oa_planes.cuh"

// largest excess of |v - digits| over that of digits from FP64 remainders, relative to |v|
static double excess(int nt, bool pair) {
  std::mt19937_64 rng(7);
  std::normal_distribution<double> nd;
  double worst = 0.0;
  for (int i = 0; i < 200000; ++i) {
    double v[2], got[2] = {0, 0};
    for (int k = 0; k < 2; ++k) v[k] = nd(rng) * std::exp2((int)(rng() % 40) - 30);
    if (pair) {
      __nv_bfloat162 h[3];
      oa_bf16_digits2(v[0], v[1], nt, h);
      for (int q = 0; q < nt; ++q) { got[0] += __low2float(h[q]); got[1] += __high2float(h[q]); }
    } else {
      for (int k = 0; k < 2; ++k) {
        __nv_bfloat16 h[3];
        oa_bf16_digits(v[k], nt, h);
        for (int q = 0; q < nt; ++q) got[k] += __bfloat162float(h[q]);
      }
    }
    for (int k = 0; k < 2; ++k) {
      double r = v[k];
      for (int q = 0; q < nt; ++q) r -= (double)__bfloat162float(__float2bfloat16_rn((float)r));
      worst = std::fmax(worst, (std::fabs(v[k] - got[k]) - std::fabs(r)) / std::fabs(v[k]));
    }
  }
  return worst;
}

int main() {
  for (int nt = 2; nt <= 3; ++nt)
    for (int pair = 0; pair < 2; ++pair) printf("%d %d %.3e\n", nt, pair, excess(nt, pair));
  return 0;
}
"""


def test_digits_keep_the_value(tmp_path):
    nvcc = build.nvcc()
    if not os.path.isabs(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "digits.cu", tmp_path / "digits"
    src.write_text(SRC)
    subprocess.run([nvcc, *build.ARCH, "-O2", "-std=c++17", "-I", build.CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = [line.split() for line in out if line]
    assert len(rows) == 4
    # both ways round the last remainder, at most 2^-16 of the value, to FP32 before its digit is taken:
    # at a boundary of that rounding they may go apart, by 2^-24 of the remainder
    for nt, pair, worst in rows:
        assert float(worst) <= 2.0 ** -40, (nt, pair, worst)
