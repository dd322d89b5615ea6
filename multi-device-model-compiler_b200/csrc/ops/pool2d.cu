// mgpuPool2d (reference: lib/Kernels/GPU/Ops.cu:342-374, CPU twin lib/Kernels/CPU/Ops.cpp:161-210).
// fp32 NCHW tensors.  One thread per output element, window read straight from global memory
// (adjacent threads read adjacent windows, so every line is fetched from HBM once and
// re-served by L1/L2).  method 0 = max over the in-bounds elements, 1 = average with the
// padding counted (divisor = window elements inside the padded extent = KH*KW for every
// window that fits).
//
// Bound by HBM bytes (input once, output once).  What kept it from them was the index arithmetic, two
// 64-bit divisions per output, and window loops of run-time length, whose loads went out one at a
// time: sizes 2, 3 and 4 are compiled in and divisions are multiplications now.  Whole call, cold:
// 384 planes of 256 x 256, max 4 x 4: 30.7 -> 24.6 us; 974 of 140 x 135, 2 x 2: 41.0 -> 26.6; 213 of
// 242 x 231, average 3 x 3, stride 3: 24.6 -> 16.4; 2113 of 57 x 46, 4 x 4, stride 2: 24.6 -> 14.4.
// Set up while the kernel ahead drains (pdl.cuh): the first of these one after another 18.4 -> 16.6 us.
#include <type_traits>

#include "fast_div.h"
#include "ops_common.h"
#include "pool_slices.h"

namespace mdc {
namespace {

struct PoolGeom {
  int H, W, OH, OW, KH, KW, PHL, PWL, PHR, PWR, SH, SW;
  int oh0;    // first output row of this launch
  int total;  // outputs of this launch: rows [oh0, oh0 + by_oh) of every plane
  Divisor by_ow, by_oh;
};

// K: window size when square and compiled in, else 0
template <bool AVG, int K>
__global__ void __launch_bounds__(256) pool2d_kernel(const float *__restrict__ x, float *__restrict__ out, const PoolGeom g) {
  pdl_launch_dependents();
  pdl_wait();
  const unsigned i = blockIdx.x * 256u + threadIdx.x;
  if (i >= static_cast<unsigned>(g.total)) return;
  const int idx = static_cast<int>(i), t = g.by_ow.div(idx), ow = g.by_ow.mod(idx, t);
  const int plane = g.by_oh.div(t), oh = g.by_oh.mod(t, plane) + g.oh0;
  const float *src = x + static_cast<int64_t>(plane) * g.H * g.W;
  const int kh_n = K ? K : g.KH, kw_n = K ? K : g.KW;
  const int ih0 = oh * g.SH - g.PHL, iw0 = ow * g.SW - g.PWL;
  float acc = AVG ? 0.f : -INFINITY;
  if (K && ih0 >= 0 && iw0 >= 0 && ih0 + K <= g.H && iw0 + K <= g.W) {
    const float *s = src + ih0 * g.W + iw0;
    float v[K ? K * K : 1];
#pragma unroll
    for (int a = 0; a < K; ++a)
#pragma unroll
      for (int b = 0; b < K; ++b) v[a * K + b] = __ldg(s + a * g.W + b);
#pragma unroll
    for (int a = 0; a < K * K; ++a) acc = AVG ? acc + v[a] : fmaxf(acc, v[a]);
  } else {
    const int ih_hi = min(ih0 + kh_n, g.H), iw_hi = min(iw0 + kw_n, g.W);
    for (int ih = max(ih0, 0); ih < ih_hi; ++ih)
      for (int iw = max(iw0, 0); iw < iw_hi; ++iw) {
        const float v = __ldg(src + ih * g.W + iw);
        acc = AVG ? acc + v : fmaxf(acc, v);
      }
  }
  if (AVG) {
    // padding counts, anything beyond the padded extent does not
    const int rows = min(ih0 + kh_n, g.H + g.PHR) - ih0;
    const int cols = min(iw0 + kw_n, g.W + g.PWR) - iw0;
    acc /= float(max(rows * cols, 1));
  }
  out[idx] = acc;
}

// Non-overlapping windows without padding whose rows are one aligned vector (KW == SW == VEC,
// W a multiple of VEC): each window row is a single 8- or 16-byte load, those of a square window in
// flight together.
template <bool AVG, int VEC>
__global__ void __launch_bounds__(256) pool2d_tiled_kernel(const float *__restrict__ x, float *__restrict__ out,
                                                           const PoolGeom g) {
  using V = typename std::conditional<VEC == 4, float4, float2>::type;
  pdl_launch_dependents();
  pdl_wait();
  const unsigned i = blockIdx.x * 256u + threadIdx.x;
  if (i >= static_cast<unsigned>(g.total)) return;
  const int idx = static_cast<int>(i), t = g.by_ow.div(idx), ow = g.by_ow.mod(idx, t);
  const int plane = g.by_oh.div(t), oh = g.by_oh.mod(t, plane) + g.oh0;
  const float *src = x + (static_cast<int64_t>(plane) * g.H + oh * g.SH) * g.W + ow * VEC;
  float acc = AVG ? 0.f : -INFINITY;
  auto take = [&](const V &v) __attribute__((always_inline)) {
    if constexpr (VEC == 4) acc = AVG ? acc + v.x + v.y + v.z + v.w : fmaxf(fmaxf(acc, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
    else acc = AVG ? acc + v.x + v.y : fmaxf(acc, fmaxf(v.x, v.y));
  };
  if (g.KH == VEC) {
    V v[VEC];
#pragma unroll
    for (int kh = 0; kh < VEC; ++kh) v[kh] = __ldcs(reinterpret_cast<const V *>(src + static_cast<int64_t>(kh) * g.W));
#pragma unroll
    for (int kh = 0; kh < VEC; ++kh) take(v[kh]);
  } else {
    for (int kh = 0; kh < g.KH; ++kh) take(__ldg(reinterpret_cast<const V *>(src + static_cast<int64_t>(kh) * g.W)));
  }
  out[idx] = AVG ? acc / float(g.KH * VEC) : acc;
}

template <bool AVG>
void launch_pool(const float *x, float *out, const PoolGeom &g, bool tiled, cudaStream_t s) {
  const unsigned grid = (static_cast<unsigned>(g.total) + 255u) / 256u;
  auto launch = [&](auto kern) { check_cuda(launch_chain(kern, dim3(grid), dim3(256), 0, s, 1, x, out, g), "launch pool2d"); };
  if (tiled && g.KW == 4) launch(pool2d_tiled_kernel<AVG, 4>);
  else if (tiled) launch(pool2d_tiled_kernel<AVG, 2>);
  else if (g.KH == 2 && g.KW == 2) launch(pool2d_kernel<AVG, 2>);
  else if (g.KH == 3 && g.KW == 3) launch(pool2d_kernel<AVG, 3>);
  else if (g.KH == 4 && g.KW == 4) launch(pool2d_kernel<AVG, 4>);
  else launch(pool2d_kernel<AVG, 0>);
}

}  // namespace
}  // namespace mdc

using namespace mdc;

MDC_API void mgpuPool2d(float *input, float *output, int64_t N, int64_t C, int64_t H, int64_t W, int64_t OH,
                        int64_t OW, int64_t KH, int64_t KW, int64_t PHL, int64_t PWL, int64_t PHR, int64_t PWR,
                        int64_t SH, int64_t SW, int64_t method, void *stream) {
  if (N <= 0 || C <= 0 || OH <= 0 || OW <= 0) return;
  if (H <= 0 || W <= 0 || KH <= 0 || KW <= 0 || SH <= 0 || SW <= 0 || PHL < 0 || PWL < 0 || PHR < 0 || PWR < 0) {
    fail("mgpuPool2d: sizes and strides must be positive, paddings non-negative");
    return;
  }
  if (method != 0 && method != 1) { fail("mgpuPool2d: method must be 0 (max) or 1 (average)"); return; }
  if ((OH - 1) * SH + KH > H + PHL + PHR || (OW - 1) * SW + KW > W + PWL + PWR) {
    fail("mgpuPool2d: output extent does not fit the padded input");
    return;
  }
  // a window that lies wholly in the padding has no defined maximum
  if (method == 0 && (PHL >= KH || PWL >= KW || (OH - 1) * SH - PHL >= H || (OW - 1) * SW - PWL >= W)) {
    fail("mgpuPool2d: a window lies entirely inside the padding");
    return;
  }
  if (H * W > INT32_MAX || OH > INT32_MAX || OW > INT32_MAX) {
    fail("mgpuPool2d: shape exceeds this library's index range");
    return;
  }
  if (!device_info().ok) return;
  PoolGeom g;
  g.H = int(H), g.W = int(W), g.OH = int(OH), g.OW = int(OW), g.KH = int(KH), g.KW = int(KW);
  g.PHL = int(PHL), g.PWL = int(PWL), g.PHR = int(PHR), g.PWR = int(PWR), g.SH = int(SH), g.SW = int(SW);
  g.by_ow = Divisor(OW);
  cudaStream_t s = as_stream(stream);
  const bool tiled = PHL == 0 && PWL == 0 && KW == SW && (KW == 4 || KW == 2) && W % KW == 0 &&
                     (OH - 1) * SH + KH <= H && OW * KW <= W &&
                     reinterpret_cast<uintptr_t>(input) % (KW * 4) == 0;
  // output indices are 31 bits
  for_each_pool_slice(N * C, OH, OW, int64_t(1) << 30, [&](const PoolSlice &p) {
    g.oh0 = int(p.row0), g.by_oh = Divisor(p.rows);
    g.total = int(p.planes * p.rows * OW);
    const float *x = input + p.plane0 * H * W;
    float *y = output + p.plane0 * OH * OW + p.row0 * OW;
    if (method == 1) launch_pool<true>(x, y, g, tiled, s);
    else launch_pool<false>(x, y, g, tiled, s);
  });
  check_cuda(cudaGetLastError(), "launch pool2d");
  launched("mdc_pool2d");
}
