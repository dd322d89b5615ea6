// Tile choice of the tensor-core Gemms.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace mdc {

struct GemmTile {
  bool one_wave = false;  // gemm_one_wave_kernel; otherwise the persistent kernel of gemm_tcgen05.cu
  int cg = 2;             // CTAs per tile (2 = tcgen05 CTA pair)
  int box_m = 128;        // rows of A per CTA, a multiple of 8
  int mma_m = 128;        // rows of its accumulator: 64 or 128
  int bn = 256;           // output columns per tile
  int depth = 1;          // 64-wide k-blocks per ring stage
  int stages = 4;
};

constexpr int kOneWaveMaxSmem = 226 * 1024;  // the rest of the 227 KiB is the kernel's static part

GemmTile choose_gemm_tile(int64_t M, int64_t N, int64_t K, int sms);

// Columns per CTA of gemm_few_rows: 16 spread a narrow weight over more SMs; 32 read whole lines of a wide one.
inline int few_rows_columns(int64_t N, int sms) { return (N + 15) / 16 <= sms ? 16 : 32; }

// Largest K that gemm_few_rows takes.  A CTA of it walks K alone, so its time grows with K and hardly with N;
// converting the weight first goes over the whole chip, and its time grows with K and N: few rows win at a short K,
// and at any K once there are columns enough for the SMs.  How many depends on how a row of W comes: in 16-byte
// vectors or value by value, and for 32 columns in whole lines or not.  us a call, calls one after another, converted /
// few rows, 16 rows, inputs out of memory:
//   16 columns, vectors      256 x 1024 6.6 / 5.2     1000 x 1536 8.1 / 6.7     1000 x 3072 11.7 / 10.3
//                            1300 x 2048 11.1 / 8.6   1800 x 3072 14.6 / 10.8   2000 x 6144 25.3 / 16.4
//                            1000 x 2048 10.5 / 8.4   1344 x 3200 13.3 / 10.7   704 x 6912 17.8 / 16.7
//   16 columns, by value     601 x 768 6.6 / 5.8      1001 x 1536 8.5 / 8.2     2001 x 1536 10.4 / 8.2
//                            2001 x 2048 11.3 / 10.3
//   32 columns, whole lines  2400 x 6144 25.2 / 25.4  2816 x 4096 19.6 / 18.3   4096 x 4096 24.9 / 19.3
//   32 columns, vectors      2600 x 1280 9.8 / 8.1    2600 x 2048 13.2 / 11.3   3700 x 3072 21.3 / 15.4
//   32 columns, by value     2369 x 1280 9.9 / 9.4    2401 x 1536 10.5 / 10.4   4401 x 3072 24.8 / 17.9
//                            with 64 rows 2369 x 768 10.2 / 8.5, x 1024 11.0 / 9.3
// Beyond one CTA per SM the second wave costs as much as the first (5000 x 1024 10.5 / 13.4, 32000 x 768 36.4 / 44.5),
// until the copy of the weight no longer stays in L2: 50257 x 768 81 / 75, 32000 x 2048 109 / 82.  A second wave
// that is at least two thirds full still wins at a short K: 7500 x 512 10.3 / 9.7, but 7008 x 512 9.3 / 9.5 and 8500 x 768 11.8 /
// 12.7.
// The lines are older than both sides of these figures and stand too early: of the calls above they convert 1000 x 3072, 1300 x
// 2048, 2000 x 6144, 704 x 6912, 2001 x 2048 and 2600 x 2048, as they do 32 x 2227 x 4354 (23.7 / 19.1) and 64 x 2828 x 8152 (43.3 /
// 34.7; but 8 x 256 x 6912 14.5 / 16.5 and 64 x 320 x 2432 8.5 / 9.6 rightly).  In the second wave they stand too late: 9001 x 512 10.4 /
// 11.0, 8 x 7500 x 640 10.4 / 11.9.
inline int64_t few_rows_max_k(int64_t M, int64_t N, bool vectors, bool lines, int sms) {
  if (few_rows_columns(N, sms) == 16) {
    if (!vectors) return std::min<int64_t>(1536, std::max<int64_t>(512, 5 * N / 4));
    if (N >= 1700) return 3 * N;
    return std::max<int64_t>(1024, N % 8 == 0 ? 5 * N / 2 : std::min<int64_t>(5 * N / 2, 1792));  // rows on sectors or not
  }
  if (lines) return 3 * N;
  if (vectors) return N >= 3700 ? 3 * N : 1280;
  return N >= 4000 ? 2 * N : M <= 32 ? 1280 : 768;
}

// Whether gemm_few_rows takes a call whose fp32 weight would have to be converted first.
// An output that overlaps the weight stays with the conversion: it has read the whole weight before the
// first store, while here CTAs still read columns of it that others have finished and stored over.
inline bool gemm_takes_few_rows(int64_t M, int64_t N, int64_t K, const float *w, const float *out, int sms) {
  if (M > 64 || N > (1 << 30) || K > (1 << 30)) return false;
  const uintptr_t w0 = reinterpret_cast<uintptr_t>(w), o0 = reinterpret_cast<uintptr_t>(out);
  if (N > 32 * sms) {
    if (K * N < 38000000 && (K > 640 || N < 50 * sms || N > 64 * sms)) return false;
  } else if (K > few_rows_max_k(M, N, N % 4 == 0 && (w0 & 15u) == 0, N % 32 == 0 && (w0 & 127u) == 0, sms)) {
    return false;
  }
  return o0 >= w0 + static_cast<uintptr_t>(K) * N * 4 || w0 >= o0 + static_cast<uintptr_t>(M) * N * 4;
}

// Whether gemm_few_rows converts the input too, every CTA for itself, instead of a launch ahead: a launch and its scratch
// less, for M * K values more that a CTA reads.  us a call, calls one after another, two launches / one, inputs out of memory:
//   K = 256, 256 columns   16 rows 6.1 / 3.7, 32 rows 6.2 / 4.6, 48 rows 6.2 / 5.7, 64 rows 6.2 / 6.7
//   K = 512, 1000 columns  16 rows 6.1 / 4.4, 32 rows 6.1 / 5.1, 48 rows 6.1 / 6.2
//   K = 768, 768 columns   16 rows 6.1 / 4.9, 32 rows 6.1 / 5.7, 48 rows 6.1 / 6.9
//   K = 1500, 2000 columns 16 rows 7.8 / 6.8, 24 rows 7.9 / 8.1
//   K = 2048, 1000 columns  8 rows 8.3 / 7.5, 16 rows 8.4 / 7.7;  K = 4096, 4096 columns 8 rows 19.3 / 18.4, 16 rows 19.3 / 18.7
//   input read value by value: 770, 500 columns 16 rows 6.3 / 5.9, 24 rows 6.3 / 7.0;  1501, 1000 columns 8 rows 7.4 / 6.7, 12 rows 7.4 / 7.2
// Up to 8 rows the launch is worth more than what the CTAs read, up to 40000 values, or 16000 that come one by one; beyond
// one CTA per SM each wave reads them again:
//   1 row   2000 x 6000 16.0 / 15.1, 4736 x 14000 59.1 / 58.0
//   8 rows  4096 x 5000 22.9 / 22.2 (40000 values), 2816 x 6000 25.3 / 25.9, 4096 x 10000 40.7 / 41.9
//   by value  4 rows  1700 x 3001 10.7 / 9.9, 2816 x 7001 28.9 / 29.8;  6 rows  1700 x 3001 10.7 / 10.6;  8 rows  2000 x 3001 10.6 / 10.3
//   two waves and more  7500 x 640 8 rows 12.8 / 11.9;  16384 x 2400 2 rows 52.2 / 52.8, 8 rows 52.2 / 53.0;  30000 x 1600 6 rows 68.7 / 70.6
// From 9 rows to 16 the line is at 1536 and from 17 to 32 at 512, where the old form of the kernel stopped winning; the present one
// still wins at 16 rows and K = 4096, and at 32 rows and K = 768 only where the host needs 6 us for two launches (5.6 / 5.4 in a
// graph).  Waves were left out of it: 16 x 50257 x 768 70.5 / 74.5.
// Below 256 nothing was measured and the launch ahead stays, as it does for an output that overlaps the input: it has read
// the input before the first store.
inline bool few_rows_convert(const float *x, const float *out, int64_t M, int64_t N, int64_t K, int sms) {
  const uintptr_t x0 = reinterpret_cast<uintptr_t>(x), o0 = reinterpret_cast<uintptr_t>(out);
  if (o0 < x0 + static_cast<uintptr_t>(M) * K * 4 && x0 < o0 + static_cast<uintptr_t>(M) * N * 4) return false;
  if (K < 256) return false;
  const bool by_value = K % 4 || (x0 & 15u);
  if (M <= 8) return M * K <= (by_value ? 16000 : 40000) / ((N + 32 * sms - 1) / (32 * sms));
  if (by_value) return M <= 16 && K <= 768;
  return (M <= 16 && K <= 1536) || (M <= 32 && K <= 512);
}

// out[M, N] = x[M, K] . w[K, N] + bias, operands rounded to fp16, the weight as the caller has it
// (gemm_few_rows_tcgen05.cu).  a16: x as fp16 [M, Kp], or null where the kernel converts it (few_rows_convert).  With a16
// it follows the launch that converts it, which lets it start after its own wait (OperandList::launch with `late`): the
// weight is read ahead of that launch's end.
void gemm_few_rows(const void *a16, const float *x, const float *w, const float *bias, float *out, int64_t M, int64_t N, int64_t K,
                   cudaStream_t s);

// One call of the one-wave kernel.  w_ready: W was complete before this launch was issued (it does
// not come from a kernel still queued), so it may be read ahead of the dependency wait.
void gemm_one_wave_launch(const GemmTile &t, const void *a, const void *w_nk, const float *bias, const void *residual,
                       void *out, int64_t M, int64_t N, int64_t Kp, int32_t dtype, int32_t out_dtype, int32_t act,
                       bool w_ready, cudaStream_t s);

}  // namespace mdc
