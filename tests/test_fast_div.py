"""Division by an invariant as a multiplication (internal.h): equal to the
integer division for all divisors up to 4096, around the powers of two and at
random, at the dividends where a wrong constant shows (CPU)."""
import os
import subprocess

import pytest

from conftest import ROOT

SRC = r"""
#include <cstdint>
#include <cstdio>
#include <random>
#include "internal.h"
int main() {
  std::mt19937_64 r(1);
  long bad = 0, n = 0;
  auto check = [&](int32_t d) {
    const er::FastDiv f = er::fast_div(d);
    auto at = [&](int64_t a) {
      if (a < 0 || a > INT32_MAX) return;
      n++;
      bad += f((int32_t)a) != (int32_t)a / d;
    };
    at(0); at(d - 1); at(d); at(INT32_MAX); at(INT32_MAX / d * (int64_t)d - 1);
    for (int k = 0; k < 50; k++) {
      const int64_t q = (int64_t)(r() % (uint64_t)(INT32_MAX / d + 1));
      at(q * d); at(q * d - 1); at(q * d + d - 1); at((int64_t)(r() & INT32_MAX));
    }
  };
  for (int32_t d = 1; d <= 4096; d++) check(d);
  for (int l = 0; l < 31; l++)
    for (int e = -2; e <= 2; e++) {
      const int64_t d = ((int64_t)1 << l) + e;
      if (d >= 1 && d <= INT32_MAX) check((int32_t)d);
    }
  for (int k = 0; k < 5000; k++) check((int32_t)(r() % INT32_MAX) + 1);
  std::printf("%ld %ld\n", bad, n);
}
"""


def test_fast_div(tmp_path):
    cuda = "/usr/local/cuda/include"
    if not os.path.isdir(cuda):
        pytest.skip("CUDA headers not found")
    src, exe = tmp_path / "d.cpp", tmp_path / "d"
    src.write_text(SRC)
    csrc = os.path.join(ROOT, "tfg-pathtracer_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + csrc, "-I" + os.path.join(ROOT, "include"), "-isystem", cuda,
                    str(src), "-o", str(exe)], check=True)
    bad, n = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and n > 1_000_000
