"""The choice of the Gemm that reads an fp32 weight itself (gemm_plan.h), compiled for the host."""
import os
import shutil
import subprocess

import pytest

OPS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multi-device-model-compiler_b200", "csrc", "ops")
CUDA_INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include "gemm_plan.h"
#include <cassert>
#include <cstdio>
using mdc::gemm_takes_few_rows;
int main() {
  static float mem[4096];
  float *w = mem + 1024;
  const int64_t M = 3, N = 20, K = 12;  // 240 floats of weight, 60 of output
  for (int64_t at = -1024; at + M * N <= 3072; ++at) {
    const bool overlap = at < K * N && at + M * N > 0;
    assert(gemm_takes_few_rows(M, N, K, w, w + at) == !overlap);
  }
  const float *far = reinterpret_cast<const float *>(uintptr_t(1) << 44);
  assert(gemm_takes_few_rows(64, 1, 1536, w, far) && !gemm_takes_few_rows(65, 1, 1, w, far));
  assert(!gemm_takes_few_rows(1, 512, 1537, w, far) && gemm_takes_few_rows(1, 516, 1537, w, far));
  assert(gemm_takes_few_rows(1, 1 << 30, 1 << 20, w, reinterpret_cast<const float *>(uintptr_t(1) << 60)));
  assert(!gemm_takes_few_rows(1, 1 << 30, 1 << 20, w, reinterpret_cast<const float *>(uintptr_t(1) << 50)));
  std::puts("ok");
}
"""


def test_few_rows_rule(tmp_path):
    if not shutil.which("g++") or not os.path.isdir(CUDA_INCLUDE):
        pytest.skip("needs a host compiler and the CUDA headers")
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", OPS, "-I", CUDA_INCLUDE, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"
