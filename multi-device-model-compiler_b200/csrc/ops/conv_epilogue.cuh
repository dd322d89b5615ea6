// What the convolution kernels do with a group of G channels of a tile, one pixel to a thread: `left` channels of the tile
// from the group's first on, pixels of a channel P values apart.  The short last group has tests per channel, a whole one none.
#pragma once

#include <cstdint>

namespace mdc {

// The group's residual, to add before the activation; unchanged beyond `left`.
template <int G>
__device__ __forceinline__ void conv_fetch(float (&extra)[G], const float *src, int P, int left) {
  if (left >= G) {
#pragma unroll
    for (int j = 0; j < G; ++j, src += P) extra[j] = __ldg(src);
  } else {
#pragma unroll
    for (int j = 0; j < G; ++j, src += P)
      if (j < left) extra[j] = __ldg(src);
  }
}

// The accumulators of the group plus bias (four at a time out of shared memory) and residual, activated.
template <int G, bool kAdd, int N>
__device__ __forceinline__ void conv_finish(uint32_t (&a)[G], const float *bias, const float (&extra)[N], bool relu) {
#pragma unroll
  for (int j = 0; j < G; j += 4) {
    float4 b = *reinterpret_cast<const float4 *>(bias + j);
    if constexpr (kAdd) b.x += extra[j], b.y += extra[j + 1], b.z += extra[j + 2], b.w += extra[j + 3];
    a[j] = __float_as_uint(__uint_as_float(a[j]) + b.x);
    a[j + 1] = __float_as_uint(__uint_as_float(a[j + 1]) + b.y);
    a[j + 2] = __float_as_uint(__uint_as_float(a[j + 2]) + b.z);
    a[j + 3] = __float_as_uint(__uint_as_float(a[j + 3]) + b.w);
  }
  if (relu) {
#pragma unroll
    for (int j = 0; j < G; ++j) a[j] = __float_as_uint(fmaxf(__uint_as_float(a[j]), 0.f));
  }
}

template <int G>
__device__ __forceinline__ void conv_store(float *dst, const uint32_t (&a)[G], int P, int left) {
  if (left >= G) {
#pragma unroll
    for (int j = 0; j < G; ++j, dst += P) *dst = __uint_as_float(a[j]);
  } else {
#pragma unroll
    for (int j = 0; j < G; ++j, dst += P)
      if (j < left) *dst = __uint_as_float(a[j]);
  }
}

}  // namespace mdc
