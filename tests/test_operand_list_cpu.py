"""The bookkeeping of the operand conversion (operand_list.h), compiled for the host."""
import os
import shutil
import subprocess

import pytest

OPS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multi-device-model-compiler_b200", "csrc", "ops")

PROGRAM = r"""
#include "operand_list.h"
#include <cassert>
#include <cstdio>
using mdc::OperandList;
int main() {
  alignas(16) static float src[64];
  alignas(16) static char dst[64];
  OperandList l;
  l.cast(src, dst, 3, 8, 8);         // contiguous: one block of 4096
  l.cast(src, dst, 300, 7, 8);       // padded: 2400 elements, blocks of 1024
  l.pack(src, dst, 65, 130);         // 2 x 3 tiles of 64
  l.cast(src + 1, dst, 513, 8, 8);   // contiguous, not aligned: element by element
  l.cast(src, dst, 0, 8, 8);         // nothing to do is not a job
  l.pack(src, dst, 4, 0);
  assert(l.n == 4 && !l.overflow);
  const long long first[4] = {0, 1, 4, 10};
  for (int i = 0; i < 4; ++i) assert(l.jobs[i].first_block == first[i]);
  assert(l.blocks == 15 && l.jobs[0].vec_ok && !l.jobs[1].vec_ok && !l.jobs[3].vec_ok);
  assert(l.jobs[2].tiles_n == 3 && l.jobs[2].pitch == 72 && !l.jobs[2].vec_ok);
  l.pack(src, dst, 8, 8);
  assert(l.n == OperandList::kMax && !l.overflow);
  const long long blocks = l.blocks;
  l.cast(src, dst, 1, 8, 8);         // one too many: remembered, so that launch() can refuse
  assert(l.overflow && l.n == OperandList::kMax && l.blocks == blocks);
  l.clear();
  assert(l.n == 0 && l.blocks == 0 && !l.overflow);
  std::puts("ok");
}
"""


def test_operand_list(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("needs a host compiler")
    src, exe = tmp_path / "list.cpp", tmp_path / "list"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", OPS, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"
