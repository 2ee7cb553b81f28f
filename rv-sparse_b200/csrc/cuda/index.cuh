// Entry indices are 32 bits and reach 2^31 - 1: sums of two of them, and an
// index past a row's end, need more.
#pragma once

#include <cstdint>

namespace rvsp {

// The middle of [lo, hi), 0 <= lo <= hi.
__host__ __device__ constexpr int32_t middle(int32_t lo, int32_t hi) {
  return lo + ((hi - lo) >> 1);
}

}  // namespace rvsp
