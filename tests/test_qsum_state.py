"""Bookkeeping of the Q sums' buffers (tmx_qsum_state.h) on the host: what counts
as laid out after a buffer could not be grown or a batch ended early."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "costuum_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "tmx_qsum_state.h"
#define CHECK(x) do { if (!(x)) { printf("%d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  TmxQsumState s;
  int grown = 0, cleared = 0, grow_rc = 0, clear_rc = 0;
  const auto lay = [&](int64_t n) {
    return s.layout(n, [&] { ++grown; return grow_rc; },
                    [&] { ++cleared; return clear_rc; });
  };
  CHECK(!s.begin());
  CHECK(lay(100) == 0 && grown == 1 && cleared == 1);
  CHECK(lay(100) == 0 && grown == 1 && cleared == 1); // a later round
  s.end();
  // a failed growth leaves nothing laid out: the earlier size starts afresh
  CHECK(!s.begin());
  grow_rc = -4;
  CHECK(lay(5000) == -4 && cleared == 1);
  CHECK(s.begin()); // (that batch did not end)
  grow_rc = 0;
  CHECK(lay(100) == 0 && grown == 3 && cleared == 2);
  s.end();
  // neither does a failed clear
  CHECK(!s.begin());
  clear_rc = -3;
  CHECK(lay(50) == -3 && s.n == -1);
  clear_rc = 0;
  CHECK(s.begin() && lay(100) == 0 && grown == 5 && cleared == 4);
  s.end();
  // counters of a batch that ended early are cleared again at the same size
  CHECK(!s.begin() && lay(100) == 0 && cleared == 4);
  CHECK(s.begin() && lay(100) == 0 && cleared == 5);
  s.end();
  CHECK(!s.begin() && lay(100) == 0 && cleared == 5);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_layout_after_failures(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
