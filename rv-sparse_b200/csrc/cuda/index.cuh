// Entry indices are 32 bits and reach 2^31 - 1: sums of two of them, and an
// index past a row's end, need more.
#pragma once

#include <cstdint>

namespace rvsp {

// The middle of [lo, hi), 0 <= lo <= hi.
__host__ __device__ constexpr int32_t middle(int32_t lo, int32_t hi) {
  return lo + ((hi - lo) >> 1);
}

// base + step < end, also where the sum is past 2^31 - 1 (the three are at
// least 0; a walk's index runs past its end by less than 2^31).
__host__ __device__ constexpr bool before(uint32_t base, uint32_t step, int32_t end) {
  return base + step < static_cast<uint32_t>(end);
}

}  // namespace rvsp
