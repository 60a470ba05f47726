// Attention of a BF16 prefill step: packed prompt rows of several requests, any number of rows a
// request. See prefill_attention.cu.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

namespace carat_b200 {

constexpr int prefill_key_tile = 128;

// Consecutive rows of one request in the step, as many as one query tile holds.
struct PrefillTile {
  int row;          // first row of the step
  int tokens;       // rows of the tile
  int position;     // logical position of the first
  int key_base;     // row of the key matrix that holds logical position 0 of this request (may be
                    // negative: positions below the window have no row)
};

// One request's rows in the step and its region of the linear staging buffer (sliding layers).
struct PrefillSegment {
  int slot;
  int first;        // logical position of its first row
  int count;
  int origin;       // logical position of the region's first row, a multiple of 128
  int stage_row;    // region's first row
  int stage_rows;   // rows of the region, a multiple of 128
};

struct PrefillAttentionArguments {
  const PrefillTile *tiles;
  int tile_count;
  int query_heads;
  int kv_heads;
  int head_dim;        // 256 or 512
  int window;          // 0 = causal over everything
  // Where key (and value) rows are: column kv_head * key_head_columns, row
  // tile.key_base + kv_head * key_head_rows + position.
  int key_head_columns;
  int key_head_rows;
  void *output;        // [rows, query_heads * head_dim] bf16
  int *device_error;
};

struct PrefillAttentionMaps {
  CUtensorMap queries;   // [rows][query heads][head_dim], box 128 query rows x 64
  CUtensorMap keys;      // 2-D, box 128 rows x 64
  CUtensorMap values;
};

// Whether the kernel takes layers of this shape: the query heads of a KV head divide a 128-row
// query tile.
inline bool prefill_attention_takes(int query_heads, int kv_heads, int head_dim) {
  return (head_dim == 256 || head_dim == 512) && kv_heads > 0 && query_heads % kv_heads == 0 &&
         128 % (query_heads / kv_heads) == 0;
}

int make_prefill_attention_maps(PrefillAttentionMaps *maps, const void *queries, int query_rows,
                                int query_heads, int kv_heads, int head_dim, const void *keys,
                                const void *values, long long key_rows, int key_columns);

int launch_prefill_attention(const PrefillAttentionMaps &maps,
                             const PrefillAttentionArguments &arguments, cudaStream_t stream);

// Sliding layers: copies the ring rows each segment's first rows still see to its staging region,
// in order of position, and clears the region's rows that nothing else writes.
struct PrefillGatherArguments {
  const PrefillSegment *segments;
  int segment_count;
  const void *key_cache;       // [slot][kv_head][capacity][head_dim] bf16
  const void *value_cache;
  void *staged_keys;           // [staging rows][kv_heads * head_dim] bf16
  void *staged_values;
  long long slot_stride;       // elements
  long long head_stride;
  int capacity;
  int window;
  int kv_heads;
  int head_dim;
};
int launch_prefill_gather(const PrefillGatherArguments &arguments, cudaStream_t stream);

// destination[to[i]] = source[from[i]] (null: i), rows of `width` bf16 values. Picks the last rows of
// the prompts that become resident, and hands their final hidden rows to the drafter's table.
int launch_copy_rows(const void *source, const int *from, void *destination, const int *to,
                     int count, int width, cudaStream_t stream);

} // namespace carat_b200
