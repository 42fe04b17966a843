"""HeldCount (csrc/heldcount.hpp): the count rises with a need, falls to what a window of steps used, and
a need that comes back doubles the window.  Built for the host with the system's C++ compiler."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SOURCE = r"""
#include "heldcount.hpp"
#include <cstdio>
#include <initializer_list>
using gmk::HeldCount;
int bad = 0;
void expect(bool ok, const char* what) { if (!ok) { std::printf("%s\n", what); ++bad; } }
int main() {
  HeldCount c;
  c.raise(2);
  expect(c.n == 2, "raise");
  c.raise(1);
  expect(c.n == 2, "raise to less");
  for (int k = 0; k < 15; ++k) expect(!c.steps(1, 1), "before the first window's end");
  expect(c.steps(0, 1) && c.n == 1, "to the window's largest need");
  c.raise(2);
  expect(c.window == 64, "a need that came back");
  for (int k = 0; k < 63; ++k) expect(!c.steps(k == 5 ? 2 : 1, 1), "window of 64");
  expect(!c.steps(1, 1) && c.n == 2, "used once in the window");
  expect(c.steps(1, 64) && c.n == 1, "counted steps");
  c.raise(3);
  c.raise(4);
  expect(c.window == 128, "one doubling for a rise in two parts");
  for (int r = 0; r < 12; ++r) { c.steps(0, 1 << 20); c.raise(4); }
  expect(c.window == 4096, "the largest window");
  HeldCount m;
  m.n = 6;
  m.least = 1;
  expect(m.steps(0, 64) && m.n == 1, "not below the least");
  expect(!m.steps(0, 64) && m.n == 1, "stays");
  HeldCount q;
  q.raise(1);
  expect(!q.steps(1, 16) && q.window == 32 && !q.steps(0, 31) && q.steps(0, 1) && q.n == 0, "the windows behind the first");
  return bad;
}
"""


def test_counts(tmp_path):
    cxx = shutil.which('g++') or shutil.which('c++')
    if cxx is None:
        pytest.skip('no host C++ compiler')
    src, exe = tmp_path / 'held.cpp', tmp_path / 'held'
    src.write_text(SOURCE)
    subprocess.run([cxx, '-std=c++17', '-I', str(ROOT / 'cfd-cylinder-flow-ghost-cell_gb300' / 'csrc'), '-o', str(exe), str(src)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
