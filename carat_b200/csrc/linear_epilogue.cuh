// Argmax epilogue of the linears: 32 accumulator columns (activation rows) of a warp's 32 features.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace carat_b200 {

__device__ __forceinline__ unsigned int orderable_bf16(float rounded) {
  // Monotonic map of a bf16-representable float to 16 bits; NaN sorts below everything, matching
  // a comparison chain that never selects NaN.
  if (rounded != rounded)
    return 0U;
  const unsigned int bits = __float_as_uint(rounded) >> 16;
  return (bits & 0x8000U) ? (~bits & 0xFFFFU) : (bits | 0x8000U);
}

// Folds the rows first_row .. row_end - 1 of the 32 columns into row_best (shared memory, one
// packed key per row of the tile, whose first row is row 0).
__device__ __forceinline__ void argmax_chunk(const uint32_t (&raw)[32], float scale, int feature,
                                             int feature_base, int output_width, int lane,
                                             int first_row, int row_end,
                                             unsigned long long *row_best) {
  unsigned long long chunk_best = 0ULL;
#pragma unroll
  for (int column = 0; column < 32; ++column) {
    const float rounded =
        __bfloat162float(__float2bfloat16_rn(__uint_as_float(raw[column]) * scale));
    // Out-of-range features lose to everything; ties inside the warp go to the lowest lane,
    // which is the lowest feature index.
    const unsigned int key =
        feature < output_width
            ? ((orderable_bf16(rounded) + 1U) << 8) | static_cast<unsigned int>(31 - lane)
            : 0U;
    const unsigned int winner = __reduce_max_sync(0xFFFFFFFFU, key);
    if (lane == column && winner != 0U) {
      const unsigned int winner_feature =
          static_cast<unsigned int>(feature_base) + (31U - (winner & 31U));
      chunk_best = (static_cast<unsigned long long>(winner >> 8) << 32) |
                   static_cast<unsigned long long>(~winner_feature);
    }
  }
  const int row = first_row + lane;
  if (row < row_end && chunk_best != 0ULL)
    atomicMax(&row_best[row], chunk_best);
}

} // namespace carat_b200
