// Division by a launch constant.
#pragma once

#include <cstdint>

namespace mdc {

// Division of numbers below 2^31 by a launch constant: q = n * mul >> shift, mul = floor(2^shift / d) + 1
// with 2^(shift - 31) >= d, so the excess of mul, at most d / 2^shift relative to 1 / d, never reaches
// the next integer.  (A run-time integer division is some 40 instructions.)
struct Divisor {
  uint32_t mul, d;
  int shift;
  explicit Divisor(int64_t v = 1) : d(static_cast<uint32_t>(v)), shift(31) {
    while ((int64_t(1) << (shift - 31)) < v) ++shift;
    mul = static_cast<uint32_t>((uint64_t(1) << shift) / static_cast<uint64_t>(v) + 1);
  }
#ifdef __CUDACC__
  __device__ __forceinline__ int div(int n) const {
    return static_cast<int>((static_cast<uint64_t>(static_cast<uint32_t>(n)) * mul) >> shift);
  }
  __device__ __forceinline__ int mod(int n, int q) const { return n - q * static_cast<int>(d); }
#endif
};

}  // namespace mdc
