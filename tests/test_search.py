"""Bisection over tour steps at the largest tours (2^31 - 2 steps), on the CPU: every
probe stays inside the bounds and the result is the first step that qualifies."""
from __future__ import annotations

import subprocess

from conftest import PKG_DIR

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "bw_search.cuh"
int main() {
  const int32_t last = 2147483645;   // 2 S - 1 of the largest tree (2^30 - 1 states)
  for (int32_t first : {0, 1, 5, 1 << 29, (1 << 30) - 1, 1 << 30, (1 << 30) + 1, last - 1, last}) {
    for (int32_t lo : {0, first / 2, first}) {
      bool in = true;
      const int32_t got = bw::first_after(lo, last, [&](int32_t x) {
        if (x < lo || x > last) { in = false; return true; }
        return x >= first;
      });
      if (!in || got != first) { std::printf("lo %d first %d: got %d\n", lo, first, got); return 1; }
    }
  }
  return 0;
}
"""


def test_largest_tour(tmp_path):
    src, exe = tmp_path / "search.cpp", tmp_path / "search"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O1", "-fwrapv", "-std=c++17", "-I", str(PKG_DIR / "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
