// How the row kernels without a row-wide reduction (GeGLU) cut a row into column ranges, one CTA
// each. Plain integer rules, so that they can be checked on the host.
#pragma once

#ifdef __CUDACC__
#define CARAT_B200_HOST_DEVICE __host__ __device__
#else
#define CARAT_B200_HOST_DEVICE
#endif

namespace carat_b200 {

constexpr int row_threads = 512;
constexpr int row_group = 8;   // columns a thread takes at a time

// Columns of every part but the last, which takes what is left: whole groups of eight columns.
CARAT_B200_HOST_DEVICE inline int row_part_columns(int width, int parts) {
  return (width / row_group + parts - 1) / parts * row_group;
}

// Parts of a GeGLU row of `width` columns (a multiple of eight). `resident`: the grid has a barrier
// and must fit the device at once (two CTAs a SM).
//  - bf16 rows, more of them than SMs: at most two column groups a thread. 2,048 rows of 21,504:
//    107 us in one part, 86 in three.
//  - otherwise two parts for wide rows while both parts of every row fit the device, where the halves
//    are equal; else one.
inline int geglu_parts(int rows, int width, bool resident, int multiprocessors) {
  if (rows > multiprocessors) {
    constexpr int most_columns = 2 * row_threads * row_group;
    return resident ? 1 : (width + most_columns - 1) / most_columns;
  }
  return width >= 8192 && width % (2 * row_group) == 0 ? 2 : 1;
}

} // namespace carat_b200
