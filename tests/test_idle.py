"""Idle things kept for reuse (tmx_idle.h) on the host: a limit for each device,
the last one put aside is taken first."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "costuum_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "tmx_idle.h"
#define CHECK(x) do { if (!(x)) { printf("%d: %s\n", __LINE__, #x); return 1; } } while (0)
static TmxIdle<int, 4, 3> idle;
int main() {
  int t = -1;
  CHECK(!idle.take(0, t) && t == -1);
  for (int i = 0; i < 4; ++i) {
    CHECK(idle.put(0, 10 + i));
  }
  CHECK(!idle.put(0, 14)); // device 0 is full, the others are not
  for (int d = 1; d < 3; ++d) {
    for (int i = 0; i < 4; ++i) {
      CHECK(idle.put(d, 20 * d + i));
    }
    CHECK(!idle.put(d, 0));
  }
  for (int d = 2; d > 0; --d) {
    for (int i = 3; i >= 0; --i) {
      CHECK(idle.take(d, t) && t == 20 * d + i);
    }
    CHECK(!idle.take(d, t));
  }
  CHECK(idle.take(0, t) && t == 13 && idle.put(0, 15) && idle.take(0, t) && t == 15);
  CHECK(!idle.put(3, 0) && !idle.put(-1, 0) && !idle.take(3, t) && !idle.take(-1, t));
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_limits_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
