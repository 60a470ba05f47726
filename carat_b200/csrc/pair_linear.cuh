// The weight-streaming linear on CTA pairs (tcgen05 cta_group::2): see pair_linear.cu.
#pragma once

#include "linear_items.cuh"

#include <cuda.h>
#include <cuda_runtime.h>

namespace carat_b200 {

constexpr int pair_features = 256;   // UMMA M of a CTA pair: output features per tile

// Activation rows of one tile (UMMA N, a multiple of 16, with e4m3 operands of 32) for a call of
// `rows` rows: one tile up to 256 rows, above that equal tiles of at most 256.
inline int pair_row_tiles(int rows) { return (rows + 255) / 256; }
inline int pair_tile_rows(int rows, int element_bytes) {
  const int granule = element_bytes == 2 ? 16 : 32;
  const int tiles = pair_row_tiles(rows);
  return ((rows + tiles - 1) / tiles + granule - 1) / granule * granule;
}

// Turns a schedule_linear() plan into one for pairs: two tiles become one, the K pieces and the
// K-cut tail stay what they are (they do not depend on the number of rows either), so every sum is
// taken in the same order in both kernels and in every batch a row can be part of. False when the
// plan's tail cannot be kept.
bool schedule_pairs(LinearPlan *plan);

// Epilogues: 0 bf16 output (K-cut tail pieces to tail_partial), 1 fp32 partial sums, 2 argmax keys.
int launch_pair_linear(const LinearPlan &plan, const KernelArguments &arguments, int mode,
                       cudaStream_t stream);

} // namespace carat_b200
