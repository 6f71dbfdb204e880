"""Remembered cluster capacities: one per device and size, and a query that
failed is asked again (host code, compiled and run here)."""
from __future__ import annotations

import os
import subprocess

PROGRAM = r"""
#include "cluster_capacity.h"
#include <cstdio>
int main() {
  b200d2::ClusterCapacity c;
  int asked = 0, answer = 0;
  auto q = [&]() { ++asked; return answer; };
  int bad = 0;
  auto expect = [&](int got, int want, const char* what) {
    if (got != want) { std::printf("%s: %d, not %d\n", what, got, want); ++bad; }
  };
  expect(c.get(0, 4, q), 1, "no answer");
  answer = 36;
  expect(c.get(0, 4, q), 36, "the answer after a failure");
  answer = 10;
  expect(c.get(0, 4, q), 36, "remembered");
  expect(asked, 2, "queries of device 0");
  expect(c.get(1, 4, q), 10, "another device");
  expect(c.get(0, 8, q), 10, "another size");
  answer = 7;
  expect(c.get(-1, 4, q), 7, "unknown device");
  expect(c.get(-1, 9, q), 7, "unknown size");
  return bad;
}
"""


def test_capacity(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src = tmp_path / "capacity.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "capacity"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(root, "t2-relion-kernel_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
