// What the convolution entry point (conv_tcgen05.cu) and the persistent kernels
// (conv_persistent_tcgen05.cu) share.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace mdc {

struct ConvShape {
  const float *x, *w, *bias, *add;
  float *out;
  int64_t N, IC, H, W, OC, KH, KW, OH, OW, PHL, PWL, SH, SW, DH, DW;
  bool relu;
};

// Whether the shape is one that the persistent kernels take.
bool conv_persistent_takes(const ConvShape &c);

// Runs the convolution on the persistent kernels; false (and nothing launched) when the shape is one
// that they do not take or there is no memory for their operands.
bool conv_persistent(const ConvShape &c, cudaStream_t s);

}  // namespace mdc
