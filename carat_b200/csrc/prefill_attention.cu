// Attention of a BF16 prefill step on tcgen05, one kernel a layer.
//
// Semantics (reference: cuda/layer_runner.cu:826-1098, causal attention with an optional sliding
// window; scale 1.0): each row attends to the keys at positions <= its own (and > its own - window).
// Scores are rounded to bf16, their softmax is fp32, probabilities are rounded to bf16 for the P.V
// product, whose fp32 sum is divided by the fp32 sum of the probabilities and rounded to bf16 once.
//
// What bounds it: a prompt row brings heads x visible keys x 4 x head_dim operations, so unlike the
// verify step's attention this is tensor-core work, and K and V come from L2 (a key is read again
// by every query tile behind it). A CTA takes 128 query rows (the query heads that share a KV head
// for 128 / heads tokens), holds Q in shared memory and walks the key tiles of 128 in order of
// position with a running maximum:
//   S = Q.K^T (128 x 128 in tensor memory, two buffers), softmax by four warps, one query row a
//   thread, P back to the same tensor-memory columns as the A operand of O += P.V.
// The tensor core computes S of the next tile while the softmax of this one runs. O (128 x 256
// fp32) takes half of tensor memory; for head_dim 512 two CTAs take 256 output components each and
// both compute S (1.5 times the work of an undivided tile, which would need all of tensor memory).
// The running maximum follows a row only when its scores outgrow it by a factor of 2^8, so O is
// seldom rescaled (lazy rescaling, a published method of recent FlashAttention kernels);
// probabilities above one cost no precision in bf16. 2,048 rows of an empty slot:
// 95 us a sliding layer (32 query heads, 16 KV heads of 256), 307 us a global one (4 of 512); in
// eight-token pieces past the first wrap a sliding layer took three launches of 4 to 10 us for
// every eight rows.
//
// Key tiles begin at multiples of 128 positions whatever the step's rows are, a tile that a row
// does not see leaves its state exactly as it was, and the decision to move the maximum is each
// row's own: a row's result depends on its position and the keys only, not on how a prompt is cut
// into steps or on the rows beside it. Sliding layers read a staging buffer in order of position
// (prefix rows gathered from the ring, new rows written beside it), global layers the cache itself.
#include "prefill_attention.cuh"

#include "context.cuh"
#include "launch.cuh"
#include "linear_items.cuh"
#include "ptx.cuh"

#include <cuda_bf16.h>
#include <math_constants.h>

namespace carat_b200 {
namespace {

constexpr int prefill_threads = 192;          // warp 0 TMA, warp 1 MMA, warps 2-5 softmax
constexpr int box_bytes = 128 * 128;          // 128 rows x 64 bf16 components
constexpr int value_boxes = 4;                // 256 output components a CTA
constexpr uint32_t output_column = 0;         // tensor memory: O 256 columns, S 2 x 128
constexpr uint32_t score_column = 256;
constexpr uint32_t tmem_columns = 512;
constexpr float log2_e = 1.4426950408889634F;
constexpr float move_threshold = 8.0F;        // in powers of two

__host__ __device__ constexpr int ring_boxes(int head_dim) { return head_dim == 256 ? 9 : 5; }

__device__ __forceinline__ float exp2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint32_t pack_bf16(float low, float high) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(low, high);
  return *reinterpret_cast<const uint32_t *>(&pair);
}

// `clears`: the key matrix is a cache, whose rows behind a tile's last token are whatever an earlier
// prompt left there, or another head's or slot's where capacity is not whole tiles. Their
// probabilities are 0, but 0 times an infinity is not: the MMA warp clears them in shared memory, in
// the last key tile of each query tile. (The staging buffer of the sliding layers is clear there.)
template <int head_dim, bool clears>
__global__ void __launch_bounds__(prefill_threads, 1)
prefill_attention_kernel(const __grid_constant__ CUtensorMap query_map,
                         const __grid_constant__ CUtensorMap key_map,
                         const __grid_constant__ CUtensorMap value_map,
                         const PrefillAttentionArguments a) {
  constexpr int key_boxes = head_dim / 64;
  constexpr int parts = head_dim / 256;
  constexpr uint32_t stages = ring_boxes(head_dim);
  constexpr uint32_t score_idesc = ptx::umma_idesc(1, 1, 128, prefill_key_tile);
  // V is the B operand read as V^T: its 64 components are the contiguous (MN) direction.
  constexpr uint32_t value_idesc = ptx::umma_idesc(1, 1, 128, 64) | (1U << 16);

  extern __shared__ unsigned char shared_raw[];
  __shared__ __align__(8) unsigned long long barriers[2 * stages + 6];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_word;

  const uint32_t query_tiles = (ptx::smem_u32(shared_raw) + 1023U) & ~1023U;
  const uint32_t ring = query_tiles + key_boxes * box_bytes;
  const uint32_t full_bar = ptx::smem_u32(&barriers[0]);
  const uint32_t empty_bar = ptx::smem_u32(&barriers[stages]);
  const uint32_t query_bar = ptx::smem_u32(&barriers[2 * stages]);
  const uint32_t score_bar = ptx::smem_u32(&barriers[2 * stages + 1]);        // two
  const uint32_t probability_bar = ptx::smem_u32(&barriers[2 * stages + 3]);  // two
  const uint32_t output_bar = ptx::smem_u32(&barriers[2 * stages + 5]);
  volatile int *abort_flag = &abort_word;

  const int warp = static_cast<int>(threadIdx.x) / 32;
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int per_tile = a.kv_heads * parts;
  const int tile_index = static_cast<int>(blockIdx.x) / per_tile;
  const int rest = static_cast<int>(blockIdx.x) - tile_index * per_tile;
  const int kv_head = rest / parts;
  const int part = rest - kv_head * parts;
  const int group = a.query_heads / a.kv_heads;

  grid_dependency_launch();
  if (threadIdx.x == 0) {
    for (uint32_t stage = 0; stage < stages; ++stage) {
      ptx::mbarrier_init(full_bar + 8U * stage, 1);
      ptx::mbarrier_init(empty_bar + 8U * stage, 1);
    }
    ptx::mbarrier_init(query_bar, 1);
    for (uint32_t buffer = 0; buffer < 2; ++buffer) {
      ptx::mbarrier_init(score_bar + 8U * buffer, 1);
      ptx::mbarrier_init(probability_bar + 8U * buffer, 4);
    }
    ptx::mbarrier_init(output_bar, 1);
    ptx::fence_mbarrier_init();
    abort_word = 0;
    ptx::prefetch_tensormap(&query_map);
    ptx::prefetch_tensormap(&key_map);
    ptx::prefetch_tensormap(&value_map);
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(&tmem_base_slot), tmem_columns);
    ptx::tmem_relinquish_alloc_permit();
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  ptx::tcgen05_fence_after_thread_sync();
  const uint32_t tmem_base = tmem_base_slot;

  // The tile list is written before the chain of dependent launches begins.
  const PrefillTile tile = a.tiles[tile_index];
  const int last = tile.position + tile.tokens - 1;
  const int lowest = a.window > 0 && tile.position >= a.window ? tile.position - a.window + 1 : 0;
  const int first_tile = lowest / prefill_key_tile;
  const int tiles = last / prefill_key_tile - first_tile + 1;

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t policy = ptx::policy_evict_last();
      uint32_t stage = 0;
      uint32_t phase = 0;
      bool healthy = true;
      grid_dependency_wait();
      ptx::mbarrier_arrive_expect_tx(query_bar, key_boxes * box_bytes);
      for (int box = 0; box < key_boxes; ++box)
        ptx::tma_load_3d(query_tiles + box * box_bytes, &query_map, box * 64, kv_head * group,
                         tile.row, query_bar, policy);
      const int key_x = kv_head * a.key_head_columns;
      const int key_y = tile.key_base + kv_head * a.key_head_rows + first_tile * prefill_key_tile;
      const auto load = [&](const CUtensorMap *map, int x, int y, int boxes) {
        for (int box = 0; box < boxes && healthy; ++box) {
          if (!ptx::mbarrier_wait_checked(empty_bar + 8U * stage, phase ^ 1U, abort_flag,
                                          a.device_error, 60)) {
            healthy = false;
            break;
          }
          ptx::mbarrier_arrive_expect_tx(full_bar + 8U * stage, box_bytes);
          ptx::tma_load_2d(ring + stage * box_bytes, map, x + box * 64, y, full_bar + 8U * stage,
                           policy);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1U;
          }
        }
      };
      // In the order the MMA warp consumes them.
      load(&key_map, key_x, key_y, key_boxes);
      for (int j = 0; j < tiles && healthy; ++j) {
        if (j + 1 < tiles)
          load(&key_map, key_x, key_y + (j + 1) * prefill_key_tile, key_boxes);
        load(&value_map, key_x + part * 256, key_y + j * prefill_key_tile, value_boxes);
      }
      if (!healthy) {
        // Copies in flight land before the CTA gives its shared memory back.
        ptx::mbarrier_wait_bounded(query_bar, 0);
        for (uint32_t other = 0; other < stages; ++other)
          ptx::mbarrier_wait_bounded(full_bar + 8U * other, other < stage ? phase : phase ^ 1U);
      }
    }
  } else if (warp == 1) {
    // The whole warp walks the loop in lockstep and one elected lane issues.
    const uint64_t key_desc = ptx::umma_desc_k_major_sw128(ring);
    const uint32_t desc_high = static_cast<uint32_t>(key_desc >> 32);
    const uint32_t ring_low = static_cast<uint32_t>(key_desc);
    const uint32_t value_low =
        static_cast<uint32_t>(ptx::umma_desc_mn_major_sw128(ring, box_bytes));
    const uint32_t query_low = static_cast<uint32_t>(ptx::umma_desc_k_major_sw128(query_tiles));
    uint32_t stage = 0;
    uint32_t phase = 0;
    bool healthy = true;
    const auto wait = [&](uint32_t bar, uint32_t parity, int code) {
      const bool ready = ptx::mbarrier_wait_checked(bar, parity, abort_flag, a.device_error, code);
      if (__all_sync(0xFFFFFFFFU, ready ? 1 : 0) == 0)
        healthy = false;
      else
        ptx::tcgen05_fence_after_thread_sync();
      return healthy;
    };
    const auto advance = [&] {
      if (++stage == stages) {
        stage = 0;
        phase ^= 1U;
      }
    };
    const auto scores = [&](int j) {
      const uint32_t accumulator = tmem_base + score_column + (j & 1) * 128;
      for (int box = 0; box < key_boxes; ++box) {
        if (!wait(full_bar + 8U * stage, phase, 61))
          return;
        if (ptx::elect_one()) {
          const uint32_t a_low = query_low + box * (box_bytes >> 4);
          const uint32_t b_low = ring_low + stage * (box_bytes >> 4);
#pragma unroll
          for (int step = 0; step < 4; ++step)
            ptx::tcgen05_mma_f16_split(accumulator, a_low + 2 * step, desc_high, b_low + 2 * step,
                                       desc_high, score_idesc, (box > 0 || step > 0) ? 1U : 0U);
          ptx::tcgen05_commit(empty_bar + 8U * stage);
        }
        __syncwarp();
        advance();
      }
      if (ptx::elect_one())
        ptx::tcgen05_commit(score_bar + 8U * (j & 1));
      __syncwarp();
    };
    if (wait(query_bar, 0, 62))
      scores(0);
    for (int j = 0; j < tiles && healthy; ++j) {
      if (j + 1 < tiles) {
        // S of the next tile goes where P of the previous one was: its product must be done.
        if (j > 0 && !wait(output_bar, (j - 1) & 1, 63))
          break;
        scores(j + 1);
        if (!healthy)
          break;
      }
      if (!wait(probability_bar + 8U * (j & 1), (j >> 1) & 1, 64))
        break;
      const uint32_t probabilities = tmem_base + score_column + (j & 1) * 128;
      for (int box = 0; box < value_boxes; ++box) {
        if (!wait(full_bar + 8U * stage, phase, 65))
          break;
        if constexpr (clears) {
          if (j + 1 == tiles) {
            // A row is 128 bytes of a box (the swizzle moves 16-byte pieces within it), four rows a
            // turn of the warp, from the box's end.
            const int unseen = (first_tile + tiles) * prefill_key_tile - (last + 1);
            const uint32_t end = ring + (stage + 1) * box_bytes;
            uint32_t address = end - 512 + lane * 16;
            const uint32_t least = end - unseen * 128;
#pragma unroll 8
            for (int turn = 0; turn < prefill_key_tile / 4; ++turn, address -= 512)
              if (address >= least)
                ptx::store_shared_zero16(address);
            ptx::fence_proxy_async();
            __syncwarp();
          }
        }
        if (ptx::elect_one()) {
          const uint32_t b_low = value_low + stage * (box_bytes >> 4);
#pragma unroll
          for (int step = 0; step < prefill_key_tile / 16; ++step)   // 16 keys = 2048 bytes of V
            ptx::tcgen05_mma_f16_tmem_a(tmem_base + output_column + box * 64,
                                        probabilities + step * 8, b_low + step * 128, desc_high,
                                        value_idesc, (j > 0 || step > 0) ? 1U : 0U);
          ptx::tcgen05_commit(empty_bar + 8U * stage);
        }
        __syncwarp();
        advance();
      }
      if (!healthy)
        break;
      if (ptx::elect_one())
        ptx::tcgen05_commit(output_bar);
      __syncwarp();
    }
  } else {
    const int quarter = warp & 3;   // TMEM lane group this warp may read
    const int row = quarter * 32 + lane;
    const int token = row / group;
    const int head = row - token * group;
    const int position = tile.position + token;
    const uint32_t lanes = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    float maximum = -CUDART_INF_F;
    float sum = 0.0F;
    bool healthy = true;
    grid_dependency_wait();
    for (int j = 0; j < tiles; ++j) {
      const uint32_t buffer = static_cast<uint32_t>(j & 1);
      const bool ready = ptx::mbarrier_wait_checked(score_bar + 8U * buffer, (j >> 1) & 1,
                                                    abort_flag, a.device_error, 66);
      if (__all_sync(0xFFFFFFFFU, ready ? 1 : 0) == 0) {
        healthy = false;
        break;
      }
      ptx::tcgen05_fence_after_thread_sync();
      const uint32_t columns = lanes + score_column + buffer * 128;
      uint32_t raw[4][32];
#pragma unroll
      for (int chunk = 0; chunk < 4; ++chunk)
        ptx::tmem_load_32x32b_x32(columns + chunk * 32, raw[chunk]);
      ptx::tmem_load_wait();
      // Scores are bf16 values, as the model defines them.
#pragma unroll
      for (int chunk = 0; chunk < 4; ++chunk)
#pragma unroll
        for (int column = 0; column < 32; column += 2) {
          const uint32_t pair = pack_bf16(__uint_as_float(raw[chunk][column]),
                                          __uint_as_float(raw[chunk][column + 1]));
          raw[chunk][column] = pair << 16;
          raw[chunk][column + 1] = pair & 0xFFFF0000U;
        }
      const int key0 = (first_tile + j) * prefill_key_tile;
      const bool whole = key0 + prefill_key_tile - 1 <= tile.position &&
                         (a.window <= 0 || key0 > last - a.window);
      if (!whole) {
        const int newest = position - key0;                                  // visible: <= newest
        const int oldest = a.window > 0 ? newest - a.window : -1;            //          > oldest
#pragma unroll
        for (int chunk = 0; chunk < 4; ++chunk)
#pragma unroll
          for (int column = 0; column < 32; ++column) {
            const int key = chunk * 32 + column;
            if (key > newest || key <= oldest)
              raw[chunk][column] = __float_as_uint(-CUDART_INF_F);
          }
      }
      float largest = __uint_as_float(raw[0][0]);
#pragma unroll
      for (int chunk = 0; chunk < 4; ++chunk)
#pragma unroll
        for (int column = 0; column < 32; ++column)
          largest = fmaxf(largest, __uint_as_float(raw[chunk][column]));
      // Move the maximum only when this tile outgrows it by more than 2^8.
      float alpha = 1.0F;
      if ((largest - maximum) * log2_e > move_threshold) {   // also from -inf to anything finite
        if (maximum != -CUDART_INF_F)
          alpha = exp2_approx((maximum - largest) * log2_e);
        maximum = largest;
      }
      if (__any_sync(0xFFFFFFFFU, alpha != 1.0F ? 1 : 0) != 0) {
        const bool done = ptx::mbarrier_wait_checked(output_bar, (j - 1) & 1, abort_flag,
                                                     a.device_error, 67);
        if (__all_sync(0xFFFFFFFFU, done ? 1 : 0) == 0) {
          healthy = false;
          break;
        }
        ptx::tcgen05_fence_after_thread_sync();
        sum *= alpha;
#pragma unroll 1
        for (int chunk = 0; chunk < 8; ++chunk) {
          uint32_t part_sums[32];
          ptx::tmem_load_32x32b_x32(lanes + output_column + chunk * 32, part_sums);
          ptx::tmem_load_wait();
#pragma unroll
          for (int column = 0; column < 32; ++column)
            part_sums[column] = __float_as_uint(__uint_as_float(part_sums[column]) * alpha);
          ptx::tmem_store_32x32b_x32(lanes + output_column + chunk * 32, part_sums);
        }
      }
      // A row that has seen nothing yet has only -inf here: exp2(-inf) = 0.
      const float offset = maximum == -CUDART_INF_F ? 0.0F : maximum * log2_e;
      float partial[4] = {0.0F, 0.0F, 0.0F, 0.0F};
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t packed[32];
#pragma unroll
        for (int pair = 0; pair < 32; ++pair) {
          const int chunk = 2 * half + pair / 16;
          const int column = (pair % 16) * 2;
          const float low =
              exp2_approx(fmaf(__uint_as_float(raw[chunk][column]), log2_e, -offset));
          const float high =
              exp2_approx(fmaf(__uint_as_float(raw[chunk][column + 1]), log2_e, -offset));
          partial[pair % 2 * 2] += low;
          partial[pair % 2 * 2 + 1] += high;
          packed[pair] = pack_bf16(low, high);
        }
        ptx::tmem_store_32x32b_x32(columns + half * 32, packed);
      }
      sum += (partial[0] + partial[1]) + (partial[2] + partial[3]);
      ptx::tmem_store_wait();
      ptx::tcgen05_fence_before_thread_sync();
      __syncwarp();
      if (lane == 0)
        ptx::mbarrier_arrive(probability_bar + 8U * buffer);
    }
    if (healthy) {
      // The product before the last may still run here, and its phase has the other parity: one
      // wait for each, or the second could take the phase before the first for its own.
      const bool done =
          (tiles < 2 || ptx::mbarrier_wait_checked(output_bar, (tiles - 2) & 1, abort_flag,
                                                   a.device_error, 68)) &&
          ptx::mbarrier_wait_checked(output_bar, (tiles - 1) & 1, abort_flag, a.device_error, 68);
      if (__all_sync(0xFFFFFFFFU, done ? 1 : 0) != 0) {
        ptx::tcgen05_fence_after_thread_sync();
        const float inverse = 1.0F / sum;
        auto *destination = static_cast<__nv_bfloat16 *>(a.output) +
                            (static_cast<size_t>(tile.row + token) * a.query_heads +
                             kv_head * group + head) *
                                head_dim +
                            part * 256;
#pragma unroll 1
        for (int chunk = 0; chunk < 8; ++chunk) {
          uint32_t raw[32];
          ptx::tmem_load_32x32b_x32(lanes + output_column + chunk * 32, raw);
          ptx::tmem_load_wait();
          if (token < tile.tokens) {
            auto *vectors = reinterpret_cast<uint4 *>(destination + chunk * 32);
#pragma unroll
            for (int vector = 0; vector < 4; ++vector) {
              uint32_t words[4];
#pragma unroll
              for (int word = 0; word < 4; ++word)
                words[word] = pack_bf16(__uint_as_float(raw[vector * 8 + word * 2]) * inverse,
                                        __uint_as_float(raw[vector * 8 + word * 2 + 1]) * inverse);
              vectors[vector] = make_uint4(words[0], words[1], words[2], words[3]);
            }
          }
        }
      }
    }
  }

  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tcgen05_fence_after_thread_sync();
    ptx::tmem_dealloc(tmem_base, tmem_columns);
  }
}

__global__ void prefill_gather_kernel(PrefillGatherArguments a) {
  grid_dependency_launch();
  const PrefillSegment segment = a.segments[blockIdx.y];
  const int before = segment.first - segment.origin;                 // prefix rows of the region
  const int end = before + segment.count;
  const int fill = before + segment.stage_rows - end;                // rows this kernel writes
  const int lowest =
      a.window > 0 && segment.first >= a.window ? segment.first - a.window + 1 : 0;
  const int row_vectors = a.kv_heads * a.head_dim / 8;
  const int head_vectors = a.head_dim / 8;
  grid_dependency_wait();
  const auto *keys = static_cast<const uint4 *>(a.key_cache);
  const auto *values = static_cast<const uint4 *>(a.value_cache);
  auto *staged_keys = static_cast<uint4 *>(a.staged_keys);
  auto *staged_values = static_cast<uint4 *>(a.staged_values);
  const long long total = static_cast<long long>(fill) * row_vectors;
  for (long long index = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
       index < total; index += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int ordinal = static_cast<int>(index / row_vectors);
    const int vector = static_cast<int>(index - static_cast<long long>(ordinal) * row_vectors);
    const int row = ordinal < before ? ordinal : end + (ordinal - before);
    const int position = segment.origin + row;
    uint4 key = make_uint4(0, 0, 0, 0);
    uint4 value = make_uint4(0, 0, 0, 0);
    if (ordinal < before && position >= lowest) {
      const int head = vector / head_vectors;
      const long long source =
          (segment.slot * a.slot_stride + head * a.head_stride) / 8 +
          static_cast<long long>(position % a.capacity) * head_vectors +
          (vector - head * head_vectors);
      key = keys[source];
      value = values[source];
    }
    const long long destination =
        static_cast<long long>(segment.stage_row + row) * row_vectors + vector;
    staged_keys[destination] = key;
    staged_values[destination] = value;
  }
}

__global__ void copy_rows_kernel(const uint4 *source, const int *from, uint4 *destination,
                                 const int *to, int vectors) {
  grid_dependency_launch();
  const int index = static_cast<int>(blockIdx.x);
  const long long first = static_cast<long long>(from != nullptr ? from[index] : index) * vectors;
  const long long last = static_cast<long long>(to != nullptr ? to[index] : index) * vectors;
  grid_dependency_wait();
  for (int vector = static_cast<int>(threadIdx.x); vector < vectors; vector += blockDim.x)
    destination[last + vector] = source[first + vector];
}

bool encode_rows(CUtensorMap *map, const void *base, long long rows, int columns) {
  const EncodeTiled encode = encode_tiled_entry();
  if (encode == nullptr || base == nullptr || rows <= 0 || columns <= 0 || columns % 8 != 0)
    return false;
  const cuuint64_t dimensions[2] = {static_cast<cuuint64_t>(columns),
                                    static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(columns) * 2};
  const cuuint32_t box[2] = {64, prefill_key_tile};
  const cuuint32_t element_strides[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dimensions,
                strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int head_dim, bool clears>
int launch_variant(const PrefillAttentionMaps &maps, const PrefillAttentionArguments &a,
                   cudaStream_t stream) {
  constexpr int dynamic_bytes = (head_dim / 64 + ring_boxes(head_dim)) * box_bytes + 1024;
  static PerDeviceOnce configured;
  if (configured.run([] {
        return cudaFuncSetAttribute(prefill_attention_kernel<head_dim, clears>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, dynamic_bytes);
      }) != cudaSuccess) {
    return -10;
  }
  const int blocks = a.tile_count * a.kv_heads * (head_dim / 256);
  return launch_chained(prefill_attention_kernel<head_dim, clears>,
                        dim3(static_cast<unsigned>(blocks)), dim3(prefill_threads), dynamic_bytes,
                        stream, false, maps.queries, maps.keys, maps.values, a) == cudaSuccess
             ? 0
             : -11;
}

} // namespace

int make_prefill_attention_maps(PrefillAttentionMaps *maps, const void *queries, int query_rows,
                                int query_heads, int kv_heads, int head_dim, const void *keys,
                                const void *values, long long key_rows, int key_columns) {
  if (maps == nullptr || queries == nullptr || query_rows <= 0 ||
      !prefill_attention_takes(query_heads, kv_heads, head_dim)) {
    return -1;
  }
  PrefillAttentionMaps result{};
  const EncodeTiled encode = encode_tiled_entry();
  if (encode == nullptr)
    return -5;
  const int group = query_heads / kv_heads;
  const cuuint64_t dimensions[3] = {static_cast<cuuint64_t>(head_dim),
                                    static_cast<cuuint64_t>(query_heads),
                                    static_cast<cuuint64_t>(query_rows)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(head_dim) * 2,
                                 static_cast<cuuint64_t>(head_dim) * 2 * query_heads};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(group),
                             static_cast<cuuint32_t>(128 / group)};
  const cuuint32_t element_strides[3] = {1, 1, 1};
  if (encode(&result.queries, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(queries),
             dimensions, strides, box, element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
      !encode_rows(&result.keys, keys, key_rows, key_columns) ||
      !encode_rows(&result.values, values, key_rows, key_columns)) {
    return -5;
  }
  *maps = result;
  return 0;
}

int launch_prefill_attention(const PrefillAttentionMaps &maps, const PrefillAttentionArguments &a,
                             cudaStream_t stream) {
  if (a.tiles == nullptr || a.tile_count <= 0 || a.output == nullptr || a.device_error == nullptr ||
      !prefill_attention_takes(a.query_heads, a.kv_heads, a.head_dim)) {
    return -1;
  }
  if (a.window > 0) {
    return a.head_dim == 256 ? launch_variant<256, false>(maps, a, stream)
                             : launch_variant<512, false>(maps, a, stream);
  }
  return a.head_dim == 256 ? launch_variant<256, true>(maps, a, stream)
                           : launch_variant<512, true>(maps, a, stream);
}

int launch_prefill_gather(const PrefillGatherArguments &a, cudaStream_t stream) {
  if (a.segments == nullptr || a.segment_count <= 0 || a.key_cache == nullptr ||
      a.value_cache == nullptr || a.staged_keys == nullptr || a.staged_values == nullptr ||
      a.capacity <= 0 || a.kv_heads <= 0 || a.head_dim % 8 != 0 || a.slot_stride % 8 != 0 ||
      a.head_stride % 8 != 0) {
    return -1;
  }
  // Two blocks a SM for a lone segment, half a block a SM and segment for several.
  const int multiprocessors = device_multiprocessors();
  const dim3 grid(a.segment_count == 1 ? 2 * multiprocessors : (multiprocessors + 1) / 2,
                  static_cast<unsigned>(a.segment_count));
  return launch_chained(prefill_gather_kernel, grid, dim3(256), 0, stream, false, a) == cudaSuccess
             ? 0
             : -11;
}

int launch_copy_rows(const void *source, const int *from, void *destination, const int *to,
                     int count, int width, cudaStream_t stream) {
  if (source == nullptr || destination == nullptr || count <= 0 || width <= 0 || width % 8 != 0)
    return -1;
  return launch_chained(copy_rows_kernel, dim3(static_cast<unsigned>(count)), dim3(256), 0, stream,
                        false, static_cast<const uint4 *>(source), from,
                        static_cast<uint4 *>(destination), to, width / 8) == cudaSuccess
             ? 0
             : -11;
}

} // namespace carat_b200
