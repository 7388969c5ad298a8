"""The divisor of a wave's pixel groups (set_divisors, internal.h) at every
wave size that the options accept: a group holds four pixels' samples, so it
can have more paths than an int counts while the wave itself does not (CPU)."""
import os
import subprocess

import pytest

from conftest import ROOT

SRC = r"""
#include <cstdint>
#include <cstdio>
#include "internal.h"
int main() {
  long bad = 0, n = 0;
  const int64_t spp[] = {1, 2, 7, 9, 4096, (1 << 24) - 1, 1 << 24, (1 << 29) - 1, 1 << 29, (1 << 29) + 1, 715827882,
                         (1 << 30) - 1, 1 << 30, (1 << 30) + 1, INT32_MAX};
  for (int64_t s : spp)
    for (int64_t npix = 1; npix <= 9 && npix * s <= INT32_MAX; npix++) {
      er::WaveParams P{};
      P.W = (int32_t)npix;
      P.H = 1;
      P.npix = (int32_t)npix;
      P.spp_wave = (int32_t)s;
      er::set_divisors(&P);
      const int64_t per = s << er::kGroup, paths = npix * s;
      const int64_t at[] = {0, 1, s - 1, s, s + 1, per - 1, per, per + 1, paths / 2, paths - 2, paths - 1};
      for (int64_t a : at) {
        if (a < 0 || a >= paths) continue;
        n++;
        bad += P.by_group((int32_t)a) != a / per;
      }
    }
  std::printf("%ld %ld\n", bad, n);
}
"""


def test_groups_of_large_waves(tmp_path):
    cuda = "/usr/local/cuda/include"
    if not os.path.isdir(cuda):
        pytest.skip("CUDA headers not found")
    src, exe = tmp_path / "g.cpp", tmp_path / "g"
    src.write_text(SRC)
    csrc = os.path.join(ROOT, "tfg-pathtracer_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + csrc, "-I" + os.path.join(ROOT, "include"), "-isystem", cuda,
                    str(src), "-o", str(exe)], check=True)
    bad, n = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0 and n > 400
