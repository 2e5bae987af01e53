"""A lane's walk over a CSR row (csrc/qs_rows.h, the code the kernels run): every entry of the row once and none outside
it, also for rows that end at the largest int32, where an int32 position plus the entries looked ahead would wrap."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qiskit-blackwell_b200", "csrc")

SOURCE = r"""
#include "qs_rows.h"
#include <cstdio>
#include <vector>
int main() {
  const int32_t top = 2147483647;
  long bad = 0, rows = 0;
  for (int V = 1; V <= 32; V *= 2)
    for (int ahead : {2, 4})
      for (int32_t end : {0, 1, 40, 100000, top - 130, top - 1, top})
        for (int32_t len : {0, 1, 2, 31, 33, 127, 128, 129, 1000}) {
          if (len > end) continue;
          ++rows;
          std::vector<int> seen(len, 0);
          for (int lane = 0; lane < V; ++lane)
            for (RowWalk w(end - len, end, lane); w.more(); w.step(V * ahead))
              for (int u = 0; u < ahead; ++u)
                if (w.has(u * V)) {
                  const int64_t k = w.at + (int64_t)u * V - (end - len);
                  if (k < 0 || k >= len) ++bad; else ++seen[k];
                }
          for (int s : seen) bad += s != 1;
        }
  printf("%ld %ld\n", rows, bad);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_walk_visits_each_entry_once(tmp_path):
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=undefined", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    rows, bad = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert int(rows) == 12 * 44 and int(bad) == 0
