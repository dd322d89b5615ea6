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
  alignas(16) static float mem[4096];
  float *w = mem + 1024;
  const int64_t M = 3, N = 20, K = 12;  // 240 floats of weight, 60 of output
  for (int64_t at = -1024; at + M * N <= 3072; ++at) {
    const bool overlap = at < K * N && at + M * N > 0;
    assert(gemm_takes_few_rows(M, N, K, w, w + at, 148) == !overlap);
  }
  alignas(128) static float far_mem[64];
  const float *out = reinterpret_cast<const float *>(uintptr_t(1) << 60), *v = far_mem;
  auto last_k = [&](int64_t M, int64_t N, const float *w) {  // the largest K taken, all shorter ones taken too
    int64_t k = 0;
    while (gemm_takes_few_rows(M, N, k + 1, w, out, 148)) ++k;
    for (int64_t longer = k + 1; longer < k + 4096; longer += 37) assert(!gemm_takes_few_rows(M, N, longer, w, out, 148));
    return k;
  };
  assert(gemm_takes_few_rows(64, 1, 512, v, out, 148) && !gemm_takes_few_rows(65, 1, 1, v, out, 148));
  // 16 columns a CTA: in vectors, off 16 bytes or an odd width value by value
  assert(last_k(1, 64, v) == 1024 && last_k(1, 600, v) == 1500 && last_k(1, 1000, v) == 2500 && last_k(1, 1300, v) == 1792);
  assert(last_k(1, 1700, v) == 5100 && last_k(1, 2368, v) == 7104 && last_k(1, 2368, v + 4) == 7104);
  assert(last_k(1, 1, v) == 512 && last_k(1, 601, v) == 751 && last_k(1, 2367, v) == 1536 && last_k(1, 2368, v + 1) == 1536);
  // 32 columns: whole lines, vectors, value by value
  assert(last_k(64, 2400, v) == 7200 && last_k(64, 2400, v + 4) == 1280 && last_k(64, 2400, v + 1) == 768);
  assert(last_k(33, 2372, v) == 1280 && last_k(33, 3700, v) == 11100 && last_k(33, 4092, v + 4) == 12276);
  assert(last_k(32, 2369, v) == 1280 && last_k(33, 2369, v) == 768 && last_k(33, 4001, v) == 8002 && last_k(1, 4736, v) == 14208);
  // more than one CTA per SM: weights that do not stay in L2
  assert(!gemm_takes_few_rows(1, 4737, 8021, v, out, 148) && gemm_takes_few_rows(1, 4737, 8022, v, out, 148));
  assert(!gemm_takes_few_rows(1, 32000, 1187, v, out, 148) && gemm_takes_few_rows(1, 32000, 1188, v, out, 148));
  // a second wave that is two thirds full
  assert(!gemm_takes_few_rows(1, 7399, 256, v, out, 148) && gemm_takes_few_rows(1, 7400, 640, v, out, 148));
  assert(!gemm_takes_few_rows(1, 7400, 641, v, out, 148) && gemm_takes_few_rows(1, 9472, 1, v, out, 148));
  assert(!gemm_takes_few_rows(1, 9473, 640, v, out, 148));
  // ranges of bytes beyond 32 bits
  assert(gemm_takes_few_rows(1, 1 << 30, 1 << 20, v, out, 148));
  assert(!gemm_takes_few_rows(1, 1 << 30, 1 << 20, v, reinterpret_cast<const float *>(uintptr_t(1) << 50), 148));
  // where the input is converted in the Gemm: rows and K, the input's alignment, no overlap with the output
  auto few_rows_convert = [](const float *x, const float *o, int64_t M, int64_t N, int64_t K) { return mdc::few_rows_convert(x, o, M, N, K, 148); };
  alignas(16) static float in[64];
  // up to 8 rows: values that all waves together read of the input
  assert(few_rows_convert(in, out, 8, 10, 5000) && !few_rows_convert(in, out, 8, 10, 5004) && few_rows_convert(in, out, 1, 4736, 14000));
  assert(few_rows_convert(in + 1, out, 8, 10, 2000) && !few_rows_convert(in + 1, out, 8, 10, 2004));
  assert(few_rows_convert(in, out, 5, 10, 3199) && !few_rows_convert(in, out, 5, 10, 3201) && !few_rows_convert(in, out, 8, 10, 1 << 20));
  assert(few_rows_convert(in, out, 8, 9472, 640) && few_rows_convert(in, out, 8, 4737, 2500) && !few_rows_convert(in, out, 8, 4737, 2504));
  assert(!few_rows_convert(in, out, 8, 1 << 30, 256) && !few_rows_convert(in, out, 6, 30000, 1600));
  assert(few_rows_convert(in, out, 16, 10, 1536) && !few_rows_convert(in, out, 16, 10, 1540) && !few_rows_convert(in, out, 17, 10, 772));
  assert(few_rows_convert(in, out, 32, 10, 512) && !few_rows_convert(in, out, 32, 10, 516) && !few_rows_convert(in, out, 33, 10, 256));
  assert(few_rows_convert(in, out, 1, 10, 256) && !few_rows_convert(in, out, 1, 10, 255));
  assert(few_rows_convert(in, out, 16, 10, 767) && !few_rows_convert(in, out, 17, 10, 767) && !few_rows_convert(in + 1, out, 16, 10, 772));
  for (int64_t at = -1024; at + 60 <= 3072; ++at)
    assert(few_rows_convert(w, w + at, 3, 20, 256) == !(at < 768 && at + 60 > 0));
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
