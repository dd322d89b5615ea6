// What the tensor-core Gemm kernels share: vector stores / residual loads of the epilogue and
// the activation arithmetic that runs beside the tensor pipe.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "activation.cuh"
#include "ptx_sm100.cuh"

namespace mdc {

// How the rows of a call can be accessed, decided on the host.
struct RowAccess {
  bool vec;   // rows of out and residual are multiples of 16 bytes, their columns of 8
  bool fast;  // and the bias can be read in 16-byte vectors
  bool wide;  // and rows can be moved 32 bytes, a whole DRAM sector, per access and thread
};
inline RowAccess row_access(int64_t N, const void *out, size_t out_elem, const void *residual, const void *bias) {
  auto al = [](const void *q, uintptr_t n) { return (reinterpret_cast<uintptr_t>(q) & (n - 1)) == 0; };
  RowAccess r;
  r.vec = N % 8 == 0 && al(out, 16) && al(residual, 16);
  r.fast = r.vec && al(bias, 16);
  r.wide = r.fast && N * static_cast<int64_t>(out_elem) % 32 == 0 && al(out, 32) &&
           (!residual || (N % 16 == 0 && al(residual, 32)));
  return r;
}

__device__ __forceinline__ void ld_global_32B(const void *src, uint32_t *r) {
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(src));
}
__device__ __forceinline__ void st_global_32B(void *dst, const uint32_t *r) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void ld_global_16B(const void *src, uint32_t *r) {
  asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "l"(src));
}
template <typename T16>
__device__ __forceinline__ uint32_t pack_pair(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack_pair<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
// 16 values of a row as TOut; dst is 32-byte aligned.  `second`: the last eight lie inside the row (a
// 16-bit row that is a multiple of 32 bytes always holds both).
template <typename TOut>
__device__ __forceinline__ void store_out16(TOut *dst, const float *v, bool second) {
  uint32_t q[16];
  if constexpr (sizeof(TOut) == 4) {
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = __float_as_uint(v[i]);
    st_global_32B(dst, q);
    if (second) st_global_32B(dst + 8, q + 8);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = pack_pair<TOut>(v[2 * i], v[2 * i + 1]);
    st_global_32B(dst, q);
  }
}
// 32 values of each lane's row (rows of a warp consecutive, row's parity the lane's; gcol a multiple of 32) as TOut, for rows of
// whole 32-byte sectors: two lanes exchange 32 bytes each and store 64 bytes of one row, then of the other.  Called by a
// whole warp.
// What bounds a large Gemm's stores is the SM's port to L2, which operands share: stores of one sector a lane leave it at
// 20 bytes a cycle, and operands, which need 64, at 15 to 40 meanwhile; sectors in pairs go at 32 (a stand-alone probe of
// eight storing warps beside bulk loads; whole lines are no faster).
template <typename TOut>
__device__ __forceinline__ void store_row_pairs(TOut *out, const float *v, int row, int M, int gcol, int N) {
  constexpr int PER = 64 / static_cast<int>(sizeof(TOut));  // values of 64 bytes
  const bool odd = threadIdx.x & 1;
  const int even_row = row & ~1;
#pragma unroll
  for (int g = 0; g < 32; g += PER) {
    uint32_t q[16], first[8], second[8];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if constexpr (sizeof(TOut) == 4) q[i] = __float_as_uint(v[g + i]);
      else q[i] = pack_pair<TOut>(v[2 * i], v[2 * i + 1]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? q[i] : q[8 + i], 1);
      first[i] = odd ? got : q[i];       // of the even lane's row
      second[i] = odd ? q[8 + i] : got;  // of the odd lane's
    }
    const int col = gcol + g + (odd ? PER / 2 : 0);
    if (col < N) {
      TOut *dst = out + static_cast<size_t>(even_row) * N + col;
      if (even_row < M) st_global_32B(dst, first);
      if (even_row + 1 < M) st_global_32B(dst + N, second);
    }
  }
}
// 8 values of a row as TOut; dst is 16-byte aligned
template <typename TOut>
__device__ __forceinline__ void store_out8(TOut *dst, const float *v) {
  if constexpr (sizeof(TOut) == 4) {
    reinterpret_cast<float4 *>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4 *>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    *reinterpret_cast<uint4 *>(dst) = make_uint4(pack_pair<TOut>(v[0], v[1]), pack_pair<TOut>(v[2], v[3]),
                                                 pack_pair<TOut>(v[4], v[5]), pack_pair<TOut>(v[6], v[7]));
  }
}
// eight 16-bit residual values (four registers) as fp32
template <typename T16>
__device__ __forceinline__ void unpack_res8(const uint32_t *r, float *v) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f;
    if constexpr (sizeof(T16) == 2 && std::is_same<T16, __half>::value)
      f = __half22float2(*reinterpret_cast<const __half2 *>(r + i));
    else
      f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(r + i));
    v[2 * i] = f.x, v[2 * i + 1] = f.y;
  }
}

// Rows that the 32-byte form does not take, NC values of which `cols` lie inside: eight at a time where
// rows allow it (vec), else one by one (static register indices).  Residuals are loaded ahead of the
// activation and of every store: loads between the stores would wait one after the other.
template <typename T16, int NC>
__device__ __forceinline__ void load_row(const T16 *res, float *rv, int cols, bool vec) {
  if (vec) {
    uint32_t r[NC / 2] = {};
#pragma unroll
    for (int g = 0; g < NC; g += 8)
      if (g < cols) ld_global_16B(res + g, r + g / 2);
#pragma unroll
    for (int g = 0; g < NC; g += 8) unpack_res8<T16>(r + g / 2, rv + g);
  } else {
#pragma unroll
    for (int j = 0; j < NC; ++j) rv[j] = j < cols ? static_cast<float>(res[j]) : 0.f;
  }
}
template <typename TOut, int NC>
__device__ __forceinline__ void store_row(TOut *out, const float *v, int cols, bool vec) {
  if (vec) {
#pragma unroll
    for (int g = 0; g < NC; g += 8)
      if (g < cols) store_out8<TOut>(out + g, v + g);
  } else {
#pragma unroll
    for (int j = 0; j < NC; ++j)
      if (j < cols) out[j] = static_cast<TOut>(v[j]);
  }
}

// Activation for the Gemm epilogue.  The epilogue runs beside the tensor pipe and must keep
// up with it; its scarce resource is the special-function unit (16 results per clock and SM,
// shared with the 16-bit conversions).  The exact-erf GELU therefore uses ONE special-function
// operation per element:
//   gelu(v) = max(v, 0) + h Phi(h),     h = max(-|v|, -8.06),     Phi(h) = 2^P(h),
// P a degree-8 polynomial fitted to log2(Phi), by its largest error weighted between the relative error of Phi and
// the absolute one of h Phi(h); beyond -8.06 h Phi(h) is below 4e-15.  A NaN stays one by the first term, +inf too, -inf becomes
// -3e-15.  Against the double-precision erf form the results of 17 million arguments are within 8.1e-7 absolute, and over [-8, 12]
// 1.3e-5 relative, an eighteenth of half an ulp of an fp16 output or less; in the 2-norm 6.5e-7 for N(0, 1) arguments.  (The
// same fit to erfc(|v| / sqrt 2) with its factors 1/2 and 1/sqrt 2 applied outside took 22 instructions a pair instead of 16 and
// was within 9.5e-7 / 1.4e-5 / 7.3e-7, +inf a NaN; the rational form of Abramowitz & Stegun 7.1.26 used before that needs a
// reciprocal as well as an exponential.)
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
using ptx::F2;
using ptx::f2;
using ptx::f2_add;
using ptx::f2_fma;
using ptx::f2_get;
using ptx::f2_mul;

__device__ __forceinline__ void gelu_erf_pair(float &va, float &vb) {
  const F2 T = f2(fmaxf(-fabsf(va), -8.0610172f), fmaxf(-fabsf(vb), -8.0610172f));
#define MDC_C2(x) f2(x, x)
  F2 P = f2_fma(MDC_C2(6.983426459328257e-08f), T, MDC_C2(3.5143536933901487e-06f));
  P = f2_fma(P, T, MDC_C2(7.777412247378379e-05f));
  P = f2_fma(P, T, MDC_C2(0.001010141335427761f));
  P = f2_fma(P, T, MDC_C2(0.008719745092093945f));
  P = f2_fma(P, T, MDC_C2(0.05425671488046646f));
  P = f2_fma(P, T, MDC_C2(-0.45826849341392517f));
  P = f2_fma(P, T, MDC_C2(1.1512970924377441f));
  P = f2_fma(P, T, MDC_C2(-0.9999945163726807f));
#undef MDC_C2
  float pa, pb;
  f2_get(P, pa, pb);
  const F2 G = f2_fma(T, f2(ex2_approx(pa), ex2_approx(pb)), f2(max_nan(va, 0.f), max_nan(vb, 0.f)));
  f2_get(G, va, vb);
}

// Applies the activation to n (even) values in place.  For rows that are stored in vectors, where the
// epilogue has to keep up with the mainloop; ragged rows, which do not, take act_apply_t: 3.7e-8
// relative (2-norm, N(0, 1) arguments) instead of 6.5e-7.
template <int ACT, int N>
__device__ __forceinline__ void act_fast_n(float *v) {
  if constexpr (ACT == kActGeluErf) {
#pragma unroll
    for (int j = 0; j < N; j += 2) gelu_erf_pair(v[j], v[j + 1]);
  } else if constexpr (ACT != kActNone) {
#pragma unroll
    for (int j = 0; j < N; ++j) v[j] = act_apply_t<ACT>(v[j]);
  }
}

}  // namespace mdc
