"""PerDevice (csrc/per_device.h), which holds the traversal kernels' grid
sizes: however many threads ask at once, each device's value is computed once
and nobody sees one in the making. Host code only, compiled here."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "oxideav-render_b200", "csrc")

PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.h"
struct Table { int first = 0, rest[7] = {}; };
int main() {
  ptd::PerDevice<Table> tables;
  std::atomic<int> fills{0}, bad{0}, ready{0};
  const Table *seen[16];
  std::vector<std::thread> th;
  for (int k = 0; k < 16; ++k)
    th.emplace_back([&, k] {
      const int device = k % 2;
      ++ready;
      while (ready < 16) {}
      std::this_thread::sleep_for(std::chrono::milliseconds(k));
      const Table &t = tables.get(device, [&](Table &t) {
        ++fills;
        t.first = device + 1;
        for (int &r : t.rest) {
          std::this_thread::sleep_for(std::chrono::milliseconds(3));
          r = device + 1;
        }
      });
      if (t.first != device + 1) ++bad;
      for (int r : t.rest) if (r != device + 1) ++bad;
      seen[k] = &t;
    });
  for (auto &t : th) t.join();
  for (int k = 2; k < 16; ++k) if (seen[k] != seen[k % 2]) ++bad;
  std::printf("%d %d\n", (int)fills, (int)bad);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_values_are_whole_and_computed_once(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split() == ["2", "0"]
