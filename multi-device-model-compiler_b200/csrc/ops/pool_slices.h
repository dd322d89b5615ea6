// How a pooling call is cut into launches whose output indices fit 31 bits: whole planes, or rows of a
// plane that alone has more than `limit` outputs.  Host arithmetic only.
#pragma once

#include <cstdint>

namespace mdc {

struct PoolSlice {
  int64_t plane0, planes, row0, rows;  // planes and output rows of one launch
};

template <typename F>
void for_each_pool_slice(int64_t planes, int64_t OH, int64_t OW, int64_t limit, F launch) {
  const int64_t per = OH * OW;
  const int64_t plane_step = per <= limit ? limit / per : 1;
  const int64_t row_step = per <= limit ? OH : (OW < limit ? limit / OW : 1);
  for (int64_t p0 = 0; p0 < planes; p0 += plane_step)
    for (int64_t r0 = 0; r0 < OH; r0 += row_step)
      launch(PoolSlice{p0, planes - p0 < plane_step ? planes - p0 : plane_step, r0, OH - r0 < row_step ? OH - r0 : row_step});
}

}  // namespace mdc
