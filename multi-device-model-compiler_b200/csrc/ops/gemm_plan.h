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

// Whether gemm_few_rows takes a call whose fp32 weight would have to be converted first.  A CTA of it walks K
// alone, at about 0.07 us per 16 values, so K is to be short or the columns many: 16 x 1000 x 2048 14.2 -> 10.5
// us, 16 x 4096 x 4096 44 -> 28 (inputs out of memory), but 16 x 1000 x 4096 25.6 -> 27.6, 16 x 491 x 2136 19.4
// -> 21.5 and 64 x 257 x 4095 25.6 -> 31.7, which stay with a conversion over the whole chip.  Rows that are not
// loaded in vectors take a shorter K still: 16 x 906 x 1751 21.5 -> 15.4, but 32 x 1221 x 3008 23.6 -> 25.6.
// An output that overlaps the weight stays with the conversion too: it has read the whole weight before the
// first store, while here CTAs still read columns of it that others have finished and stored over.
inline bool gemm_takes_few_rows(int64_t M, int64_t N, int64_t K, const float *w, const float *out) {
  if (M > 64 || N > (1 << 30) || K > (1 << 30) || (K > 1536 && K > (N % 4 == 0 ? 3 : 2) * N)) return false;
  const uintptr_t w0 = reinterpret_cast<uintptr_t>(w), o0 = reinterpret_cast<uintptr_t>(out);
  return o0 >= w0 + static_cast<uintptr_t>(K) * N * 4 || w0 >= o0 + static_cast<uintptr_t>(M) * N * 4;
}

// out[M, N] = a16[M, Kp] . w[K, N] + bias, fp16 operands, the weight as the caller has it
// (gemm_few_rows_tcgen05.cu).  It follows the launch that converts a16, which lets it start after its own
// wait (OperandList::launch with `late`): the weight is read ahead of that launch's end.
void gemm_few_rows(const void *a16, const float *w, const float *bias, float *out, int64_t M, int64_t N, int64_t K, cudaStream_t s);

// One call of the one-wave kernel.  w_ready: W was complete before this launch was issued (it does
// not come from a kernel still queued), so it may be read ahead of the dependency wait.
void gemm_one_wave_launch(const GemmTile &t, const void *a, const void *w_nk, const float *bias, const void *residual,
                       void *out, int64_t M, int64_t N, int64_t Kp, int32_t dtype, int32_t out_dtype, int32_t act,
                       bool w_ready, cudaStream_t s);

}  // namespace mdc
