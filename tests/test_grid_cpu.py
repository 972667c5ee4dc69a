"""Grids of kernels whose blocks wait for each other: as many blocks as a device
or partition holds, whatever its size, and a register count that covers the
vector.  The rules are compiled from the header that the library uses, with a
launch that refuses more blocks than fit."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include "tm_grid.h"
int main() {
  // 0 launched, 1 more than fit, 2 another error
  for (int want = 1; want <= 296; ++want)
    for (int fit = 1; fit <= 300; ++fit) {
      int blocks = want, launched = 0, calls = 0;
      const int a = tmg::launch_as_fits(blocks, 1, [&](int b) {
        ++calls;
        if (b < 1 || b > want) return 2;
        if (b > fit) return 1;
        launched = b;
        return 0;
      });
      const int most = want < fit ? want : fit;
      if (a != 0 || launched != blocks || blocks > most || blocks < most - most / 8 - 1) return 1;
      if (want <= fit && (calls != 1 || blocks != want)) return 2;
    }
  int blocks = 296, calls = 0;
  if (tmg::launch_as_fits(blocks, 1, [&](int) { ++calls; return 2; }) != 2 || calls != 1 || blocks != 296) return 3;
  blocks = 5;
  if (tmg::launch_as_fits(blocks, 1, [](int) { return 1; }) != 1 || blocks != 1) return 4;
  for (long long t = 256; t <= 75776; t += 256)
    for (long long n = 1; n <= 10 * t; n += t / 2 - 1) {
      const int e = tmg::elements_held(n, t);
      if (e == 0 ? n <= 8 * t : (e * t < n || (e > 1 && e / 2 * t >= n))) return 5;
    }
  puts("ok");
  return 0;
}
"""


def test_blocks_fit_and_cover(tmp_path):
    src, exe = tmp_path / "grid.cpp", tmp_path / "grid"
    src.write_text(SRC)
    inc = os.path.join(ROOT, "trimem_gb300", "csrc")
    try:
        subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", inc, str(src), "-o", str(exe)], check=True)
    except FileNotFoundError:
        pytest.skip("no g++")
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.returncode
