"""CPU: how often the arena's top is read back.  The bound of a graph whose rows
hold a steady part of the arena grows by 8 entries per arc and falls back with
every readback, which arrives some batches after it was asked for.  Compiled
from the header that the library uses."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "arena_room.h"
int main(int argc, char** argv) {
  const uint64_t cap = 1ull << 22, rows = strtoull(argv[1], 0, 10), ops = strtoull(argv[2], 0, 10);
  const int late = atoi(argv[3]), batches = 2000;
  const uint64_t steady = vxh::arena_bound_from(8 * rows, rows), add = 16 * ops + 8;
  uint64_t bound = steady, read = 0, since = 0;
  int asks = 0, over = 0, wait = -1;
  for (int t = 0; t < batches; ++t) {
    if (wait == 0) { read = steady; bound = read + since; }
    if (wait >= 0) --wait;
    if (bound + add > cap) ++over;
    else if (wait < 0 && vxh::arena_ask_due(bound + add, read, cap)) { ++asks; wait = late; since = 0; }
    bound += add;
    since += add;
  }
  printf("%d %d\n", asks, over);
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="needs g++")
def test_steady_rows_ask_seldom(tmp_path):
    src, exe = tmp_path / "room.cpp", tmp_path / "room"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-I" + os.path.join(ROOT, "velographx_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    cap = 1 << 22
    for rows in (1000, 100_000, 180_000, 250_000, 300_000):
        for ops in (1, 64, 475, 1000):
            for late in (0, 1, 5):
                asks, over = map(int, subprocess.run([str(exe), str(rows), str(ops), str(late)], check=True,
                                                     capture_output=True, text=True).stdout.split())
                # every readback frees at least half of the room left above the steady rows
                half = (cap - 12 * rows) / 2
                assert over == 0
                assert asks <= 2 + 2000 * (16 * ops + 8) / half, (rows, ops, late, asks)
