// Tile choice of the tensor-core Gemms.
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace mdc {

struct GemmTile {
  bool one_wave = false;  // gemm_one_wave_kernel; otherwise the persistent kernel of gemm_tcgen05.cu
  int cg = 2;             // CTAs per tile (2 = tcgen05 CTA pair)
  int box_m = 128;        // rows of A per CTA
  int bn = 256;           // output columns per tile
  int depth = 1;          // 64-wide k-blocks per ring stage
  int stages = 4;
};

constexpr int kOneWaveMaxSmem = 226 * 1024;  // the rest of the 227 KiB is the kernel's static part

GemmTile choose_gemm_tile(int64_t M, int64_t N, int64_t K, int sms);

// One call of the one-wave kernel.  w_ready: W was complete before this launch was issued (it does
// not come from a kernel still queued), so it may be read ahead of the dependency wait.
void gemm_one_wave_launch(const GemmTile &t, const void *a, const void *w_nk, const float *bias, const void *residual,
                       void *out, int64_t M, int64_t N, int64_t Kp, int32_t dtype, int32_t out_dtype, int32_t act,
                       bool w_ready, cudaStream_t s);

}  // namespace mdc
