"""How a pooling call is cut into launches (pool_slices.h), compiled for the host with small limits: the
real one, 2^30 outputs, is out of a test's reach."""
import os
import shutil
import subprocess

import pytest

OPS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multi-device-model-compiler_b200", "csrc", "ops")

PROGRAM = r"""
#include "pool_slices.h"
#include <cstdio>
#include <vector>
int main() {
  for (int64_t planes : {1, 2, 5, 7})
    for (int64_t OH : {1, 3, 8})
      for (int64_t OW : {1, 4, 9})
        for (int64_t limit : {1, 3, 4, 9, 10, 24, 35, 36, 72, 1000}) {
          std::vector<int> seen(planes * OH * OW, 0);
          mdc::for_each_pool_slice(planes, OH, OW, limit, [&](const mdc::PoolSlice &s) {
            const int64_t total = s.planes * s.rows * OW;
            // within the limit, except for a single row that is longer than it
            if (total > limit && !(s.planes == 1 && s.rows == 1)) std::printf("too large %ld\n", long(total));
            // output index within a launch: rows of a plane are contiguous, planes only when whole
            if (s.planes > 1 && s.rows != OH) std::printf("partial planes\n");
            for (int64_t i = 0; i < total; ++i) {
              const int64_t ow = i % OW, r = i / OW % s.rows, p = i / OW / s.rows;
              ++seen[((s.plane0 + p) * OH + s.row0 + r) * OW + ow];
              if (s.plane0 * OH * OW + s.row0 * OW + i != ((s.plane0 + p) * OH + s.row0 + r) * OW + ow) std::printf("wrong place\n");
            }
          });
          for (int n : seen)
            if (n != 1) std::printf("output written %d times\n", n);
        }
  std::puts("ok");
}
"""


def test_slices_cover_every_output_once(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("needs a host compiler")
    src, exe = tmp_path / "slices.cpp", tmp_path / "slices"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", OPS, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"
