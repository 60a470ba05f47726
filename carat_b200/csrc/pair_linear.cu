// Weight-streaming linear on CTA pairs (e4m3 or bf16 operands -> fp32 -> bf16).
//
// Contract (reference: cuda/linear.cu:534-803 Bf16Linear::run, Fp8Linear::run with tensor scaling):
//   output[rows, N] = bf16( scale * X[rows, K] . W[N, K]^T ), fp32 accumulation.
//
// Up to 256 rows the problem is HBM-bound, so it is a weight stream with swapped operands: output
// features are the UMMA M dimension, activation rows (padded to 16 or 32) its N dimension. Two SMs work
// on one tile of 256 features: each CTA of a pair streams its own 128 weight rows and HALF of the
// activation rows, and one tcgen05.mma of the pair (M = 256) reads both halves. Against one CTA
// per 128 features that halves the activation bytes each SM fetches from L2, writes to shared
// memory and feeds to its tensor core; what is saved there holds weights in flight instead.
// Above 256 rows (BF16 prefill) the same kernel is an ordinary tiled GEMM: the row tiles of a
// feature tile are dealt to neighbouring pairs, so its weights come from HBM once and then from L2.
// 2,048 bf16 rows: 5376 -> 43008 597 us (1.59 PFLOP/s), 21504 -> 5376 313 us with the fp32 pieces
// (1.51), 5376 -> 16384 223 us (1.62); 256 rows of 5376 -> 43008 103 us, 119 on single CTAs.
//
// The kernel stands outside the chain of programmatic dependent launches: it neither starts before
// the previous grid has ended nor lets the next one start before it has. Inside the chain, between
// grids of thousands of small CTAs, launches stopped making progress once in a few thousand; why is
// not known. (Launch order alone does not explain it: a dependent grid is admitted only when every
// CTA of the one before it has started.) What reading found is an arrival that nothing waited for:
// the commits that free the last ring stages arrive in the peer CTA too, and its only reason to stay
// was the later commit of the accumulator. An arrival that comes after the peer has left lands in
// the shared memory of whatever CTA runs there next, which inside the chain is already set up. Both
// producers now wait for the last use of every stage before the pair parts. The overlap is worth
// one to two microseconds of a launch of 40 to 600.
//
// Roles per CTA: warp 0 requests tiles by TMA (no multicast; both CTAs' copies complete on the
// leader's barrier), warp 1 of the leader issues the MMAs, warps 2-5 of both finish their 128
// features x rows from their own tensor memory. Two accumulators, so a tile's epilogue overlaps
// the next tile's loads.
#include "pair_linear.cuh"

#include "context.cuh"
#include "launch.cuh"
#include "linear_epilogue.cuh"
#include "ptx.cuh"

#include <cuda_bf16.h>

namespace carat_b200 {
namespace {

constexpr int block_bytes = 128;      // K bytes of one 128-byte swizzle atom
constexpr int pair_threads = 192;
constexpr int weight_bytes = 128 * block_bytes;
constexpr int most_stages = 10;
constexpr int ring_budget = 208 * 1024;

struct PairShape {
  int tile_rows;       // UMMA N
  int row_tiles;
  int stages;
  int tmem_columns;    // both accumulators
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  return rank;
}

__device__ __forceinline__ uint32_t in_leader(uint32_t shared_address) {
  uint32_t mapped;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(mapped) : "r"(shared_address));
  return mapped;
}

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}

__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void arrive_in_cluster(uint32_t mapped_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapped_bar)
               : "memory");
}

// Tile load into this CTA's shared memory whose completion is counted on a barrier of either CTA.
__device__ __forceinline__ void pair_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y,
                                             uint32_t mapped_bar, uint64_t policy) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global"
               ".mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::
                   "r"(dst),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(mapped_bar), "l"(policy)
               : "memory");
}

// Arrives on the barrier at this offset in both CTAs once the pair's MMAs so far have completed.
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster"
               ".multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}

template <bool wide>
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint32_t a_low, uint32_t a_high,
                                         uint32_t b_low, uint32_t b_high, uint32_t idesc,
                                         uint32_t accumulate) {
  if constexpr (wide) {
    asm volatile("{\n\t"
                 ".reg .pred p;\n\t"
                 ".reg .b64 da, db;\n\t"
                 "setp.ne.b32 p, %6, 0;\n\t"
                 "mov.b64 da, {%1, %2};\n\t"
                 "mov.b64 db, {%3, %4};\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, p;\n\t"
                 "}" ::"r"(tmem_d),
                 "r"(a_low), "r"(a_high), "r"(b_low), "r"(b_high), "r"(idesc), "r"(accumulate)
                 : "memory");
  } else {
    asm volatile("{\n\t"
                 ".reg .pred p;\n\t"
                 ".reg .b64 da, db;\n\t"
                 "setp.ne.b32 p, %6, 0;\n\t"
                 "mov.b64 da, {%1, %2};\n\t"
                 "mov.b64 db, {%3, %4};\n\t"
                 "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], da, db, %5, p;\n\t"
                 "}" ::"r"(tmem_d),
                 "r"(a_low), "r"(a_high), "r"(b_low), "r"(b_high), "r"(idesc), "r"(accumulate)
                 : "memory");
  }
}

// One feature's values of up to 32 rows, `pitch` elements apart. The whole-chunk case carries no
// predicates, so its 32 stores leave back to back.
template <typename Value, typename Convert>
__device__ __forceinline__ void store_column(const uint32_t (&raw)[32], Value *destination,
                                             uint32_t pitch, int rows, Convert convert) {
  if (rows >= 32) {
#pragma unroll
    for (uint32_t row = 0; row < 32; ++row)
      destination[row * pitch] = convert(raw[row]);
  } else {
#pragma unroll
    for (uint32_t row = 0; row < 32; ++row)
      if (static_cast<int>(row) < rows)
        destination[row * pitch] = convert(raw[row]);
  }
}

template <int mode, bool wide>
__global__ void __launch_bounds__(pair_threads, 1)
pair_linear_kernel(const __grid_constant__ CUtensorMap weight_map,
                   const __grid_constant__ CUtensorMap input_map, const KernelArguments args,
                   const PairShape shape) {
  extern __shared__ unsigned char shared_raw[];
  __shared__ __align__(8) unsigned long long barriers[2 * most_stages + 4];
  __shared__ uint32_t tmem_base_slot;
  __shared__ unsigned long long row_best[mode == 2 ? 256 : 1];

  const uint32_t input_bytes = static_cast<uint32_t>(shape.tile_rows) * (block_bytes / 2);
  const uint32_t stages = static_cast<uint32_t>(shape.stages);
  const uint32_t weight_tiles = (ptx::smem_u32(shared_raw) + 1023U) & ~1023U;
  const uint32_t input_tiles = weight_tiles + stages * weight_bytes;
  const uint32_t full_bar = ptx::smem_u32(&barriers[0]);
  const uint32_t empty_bar = ptx::smem_u32(&barriers[most_stages]);
  const uint32_t acc_full_bar = ptx::smem_u32(&barriers[2 * most_stages]);
  const uint32_t acc_empty_bar = ptx::smem_u32(&barriers[2 * most_stages + 2]);

  const int warp = static_cast<int>(threadIdx.x) / 32;
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const uint32_t rank = cluster_rank();
  const int items = item_count(args) * shape.row_tiles;
  const int first_item = static_cast<int>(blockIdx.x) / 2;
  const int item_stride = static_cast<int>(gridDim.x) / 2;

  if (threadIdx.x == 0) {
    for (uint32_t stage = 0; stage < stages; ++stage) {
      ptx::mbarrier_init(full_bar + 8U * stage, 1);
      ptx::mbarrier_init(empty_bar + 8U * stage, 1);
    }
    for (uint32_t buffer = 0; buffer < 2; ++buffer) {
      ptx::mbarrier_init(acc_full_bar + 8U * buffer, 1);
      ptx::mbarrier_init(acc_empty_bar + 8U * buffer, 8);   // four epilogue warps of each CTA
    }
    ptx::fence_mbarrier_init();
    ptx::prefetch_tensormap(&weight_map);
    ptx::prefetch_tensormap(&input_map);
  }
  if constexpr (mode == 2) {
    for (int row = static_cast<int>(threadIdx.x); row < 256; row += pair_threads)
      row_best[row] = 0ULL;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     ptx::smem_u32(&tmem_base_slot)),
                 "r"(static_cast<uint32_t>(shape.tmem_columns))
                 : "memory");
    // No relinquish of the allocation permit: it would act for the pair, and could overtake the
    // other CTA's allocation. Nothing waits for it: every other kernel here with tensor memory asks
    // for more shared memory than this one leaves, so none is on the SM beside it.
  }
  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  cluster_arrive();
  cluster_wait();   // both CTAs' barriers exist before either signals them
  ptx::tcgen05_fence_after_thread_sync();
  const uint32_t tmem_base = tmem_base_slot;
  const uint32_t accumulator_columns = static_cast<uint32_t>(shape.tmem_columns) / 2;

  if (warp == 0) {
    if (lane == 0) {
      const uint64_t stream_policy = ptx::policy_evict_first();
      const uint64_t reuse_policy = ptx::policy_evict_last();
      const uint64_t weight_policy = shape.row_tiles > 1 ? reuse_policy : stream_policy;
      const uint32_t leader_full = in_leader(full_bar);
      const uint32_t pair_bytes = 2U * (weight_bytes + input_bytes);
      const int weight_row = static_cast<int>(rank) * 128;
      const int input_row = static_cast<int>(rank) * (shape.tile_rows / 2);
      uint32_t stage = 0;
      uint32_t phase = 0;
      bool healthy = true;
      for (int index = first_item; index < items && healthy; index += item_stride) {
        const int unit = shape.row_tiles == 1 ? index : index / shape.row_tiles;
        const WorkItem item = decode_item(args, unit);
        const int y_weight = item.tile * pair_features + weight_row;
        const int y_input = (index - unit * shape.row_tiles) * shape.tile_rows + input_row;
        int k_byte = item.k_begin * block_bytes;
        for (int block = 0; block < item.k_count; ++block, k_byte += block_bytes) {
          if (!ptx::mbarrier_wait_fast(empty_bar + 8U * stage, phase ^ 1U)) {
            healthy = false;
            atomicExch(args.device_error, 1);
            break;
          }
          const uint32_t full = leader_full + 8U * stage;
          if (rank == 0)
            ptx::mbarrier_arrive_expect_tx(full_bar + 8U * stage, pair_bytes);
          pair_load_2d(weight_tiles + stage * weight_bytes, &weight_map, k_byte, y_weight, full,
                       weight_policy);
          pair_load_2d(input_tiles + stage * input_bytes, &input_map, k_byte, y_input, full,
                       reuse_policy);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1U;
          }
        }
      }
      if (healthy) {
        // The commits that free a stage arrive in both CTAs, and this CTA may not leave before the
        // last of them has: wait until each stage could be filled again.
        uint32_t tail = stage;
        uint32_t tail_phase = phase;
        for (uint32_t turn = 0; turn < stages && healthy; ++turn) {
          if (!ptx::mbarrier_wait_fast(empty_bar + 8U * tail, tail_phase ^ 1U)) {
            healthy = false;
            atomicExch(args.device_error, 1);
          }
          if (++tail == stages) {
            tail = 0;
            tail_phase ^= 1U;
          }
        }
      }
      if (!healthy && rank == 0) {
        // Let copies already in flight land before the pair gives its shared memory back: wait
        // for the phase each stage was last armed for (the other CTA waits at the cluster
        // barrier below until this one is through).
        for (uint32_t other = 0; other < stages; ++other)
          ptx::mbarrier_wait_bounded(full_bar + 8U * other, other < stage ? phase : phase ^ 1U);
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // The whole warp walks the loop in lockstep and one elected lane issues for the pair.
      const uint64_t weight_desc = ptx::umma_desc_k_major_sw128(weight_tiles);
      const uint64_t input_desc = ptx::umma_desc_k_major_sw128(input_tiles);
      const uint32_t desc_high = static_cast<uint32_t>(weight_desc >> 32);
      const uint32_t weight_low = static_cast<uint32_t>(weight_desc);
      const uint32_t input_low = static_cast<uint32_t>(input_desc);
      const uint32_t idesc =
          ptx::umma_idesc(wide ? 1U : 0U, wide ? 1U : 0U, pair_features,
                          static_cast<uint32_t>(shape.tile_rows));
      uint32_t stage = 0;
      uint32_t phase = 0;
      uint32_t buffer = 0;
      uint32_t buffer_phase = 0;
      bool healthy = true;
      for (int index = first_item; index < items && healthy; index += item_stride) {
        const WorkItem item =
            decode_item(args, shape.row_tiles == 1 ? index : index / shape.row_tiles);
        const bool free_accumulator =
            ptx::mbarrier_wait_fast(acc_empty_bar + 8U * buffer, buffer_phase ^ 1U);
        if (__all_sync(0xFFFFFFFFU, free_accumulator ? 1 : 0) == 0) {
          if (lane == 0)
            atomicExch(args.device_error, 4);
          break;
        }
        ptx::tcgen05_fence_after_thread_sync();
        const uint32_t accumulator = tmem_base + buffer * accumulator_columns;
        for (int block = 0; block < item.k_count; ++block) {
          const bool ready = ptx::mbarrier_wait_fast(full_bar + 8U * stage, phase);
          if (__all_sync(0xFFFFFFFFU, ready ? 1 : 0) == 0) {
            healthy = false;
            if (lane == 0)
              atomicExch(args.device_error, 2);
            break;
          }
          ptx::tcgen05_fence_after_thread_sync();
          const uint32_t a_low = weight_low + stage * (weight_bytes >> 4);
          const uint32_t b_low = input_low + stage * (input_bytes >> 4);
          if (ptx::elect_one()) {
            // +32 bytes along K inside the swizzle atom = +2 in the 16-byte address field.
            pair_mma<wide>(accumulator, a_low, desc_high, b_low, desc_high, idesc,
                           block > 0 ? 1U : 0U);
#pragma unroll
            for (int step = 1; step < 4; ++step)
              pair_mma<wide>(accumulator, a_low + 2 * step, desc_high, b_low + 2 * step, desc_high,
                             idesc, 1U);
            pair_commit(empty_bar + 8U * stage);
          }
          __syncwarp();
          if (++stage == stages) {
            stage = 0;
            phase ^= 1U;
          }
        }
        if (healthy && ptx::elect_one())
          pair_commit(acc_full_bar + 8U * buffer);
        __syncwarp();
        buffer ^= 1U;
        if (buffer == 0)
          buffer_phase ^= 1U;
      }
    }
  } else {
    const int quarter = warp & 3;  // TMEM lane group this warp may read
    [[maybe_unused]] const int epilogue_thread = (warp - 2) * 32 + lane;
    const uint32_t leader_acc_empty = in_leader(acc_empty_bar);
    float scale = 1.0F;
    if constexpr (mode != 1 && !wide)
      scale = args.input_scale[0] * args.weight_scale[0];
    int local = 0;
    for (int index = first_item; index < items; index += item_stride, ++local) {
      const int unit = shape.row_tiles == 1 ? index : index / shape.row_tiles;
      const WorkItem item = decode_item(args, unit);
      const int first_row = (index - unit * shape.row_tiles) * shape.tile_rows;
      const int tile_end = min(args.rows, first_row + shape.tile_rows);
      const uint32_t buffer = static_cast<uint32_t>(local & 1);
      const uint32_t use = static_cast<uint32_t>(local >> 1);
      const bool ready =
          __all_sync(0xFFFFFFFFU,
                     ptx::mbarrier_wait_bounded(acc_full_bar + 8U * buffer, use & 1U) ? 1 : 0) != 0;
      if (!ready) {
        if (lane == 0)
          atomicExch(args.device_error, 3);
        break;
      }
      ptx::tcgen05_fence_after_thread_sync();
      const int feature_base =
          item.tile * pair_features + static_cast<int>(rank) * 128 + quarter * 32;
      const int feature = feature_base + lane;
      const uint32_t lane_address = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                    buffer * accumulator_columns;
      // Where this item's sums go: fp32 pieces, or the finished rows.
      float *pieces = nullptr;
      size_t piece_width = 0;
      if constexpr (mode == 1) {
        piece_width = static_cast<size_t>(args.output_width);
        pieces = args.partial + static_cast<size_t>(item.piece) * args.rows * piece_width + feature;
      } else if constexpr (mode == 0) {
        if (item.tail) {
          const int tail_column = (args.tiles - args.tail_tiles) * pair_features;
          piece_width = static_cast<size_t>(args.output_width - tail_column);
          pieces = args.tail_partial + static_cast<size_t>(item.piece) * args.rows * piece_width +
                   (feature - tail_column);
        }
      }
#pragma unroll 1
      for (int base = first_row; base < tile_end; base += 32) {   // warp-uniform
        uint32_t raw[32];
        ptx::tmem_load_32x32b_x32(lane_address + (base - first_row), raw);
        ptx::tmem_load_wait();
        if constexpr (mode == 2) {
          argmax_chunk(raw, scale, feature, feature_base, args.output_width, lane, base, tile_end,
                       row_best);
        } else {
          if (feature < args.output_width) {
            if (mode == 1 || pieces != nullptr) {
              store_column(raw, pieces + static_cast<size_t>(base) * piece_width,
                           static_cast<uint32_t>(piece_width), tile_end - base,
                           [](uint32_t value) { return __uint_as_float(value); });
            } else {
              store_column(raw, args.output + static_cast<size_t>(base) * args.output_width + feature,
                           static_cast<uint32_t>(args.output_width), tile_end - base,
                           [scale](uint32_t value) {
                             return __float2bfloat16_rn(__uint_as_float(value) * scale);
                           });
            }
          }
        }
      }
      // The accumulator is free again as soon as its values are in registers.
      ptx::tcgen05_fence_before_thread_sync();
      __syncwarp();
      if (lane == 0)
        arrive_in_cluster(leader_acc_empty + 8U * buffer);
    }
    if constexpr (mode == 2) {
      // Every tile of this CTA is in row_best: one global atomic per row and CTA (see fp8_linear.cu).
      asm volatile("bar.sync 1, 128;" ::: "memory");
      for (int row = epilogue_thread; row < args.rows; row += 128) {
        const unsigned long long candidate = row_best[row];
        if (candidate != 0ULL)
          atomicMax(args.best + row, candidate);
      }
    }
  }

  ptx::tcgen05_fence_before_thread_sync();
  __syncthreads();
  cluster_arrive();
  cluster_wait();   // neither CTA signals the other, nor reads its operands, after this
  if (warp == 1) {
    ptx::tcgen05_fence_after_thread_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(shape.tmem_columns))
                 : "memory");
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();   // the pair's tensor memory is freed by both before either leaves
}

template <int mode, bool wide>
int launch_pairs(const LinearPlan &plan, const KernelArguments &arguments, cudaStream_t stream) {
  PairShape shape{};
  shape.tile_rows = pair_tile_rows(plan.rows, plan.element_bytes);
  shape.row_tiles = pair_row_tiles(plan.rows);
  if (mode == 2 && shape.row_tiles > 1)
    return -12;
  const int stage_bytes = weight_bytes + shape.tile_rows * (block_bytes / 2);
  shape.stages = ring_budget / stage_bytes < most_stages ? ring_budget / stage_bytes : most_stages;
  // Two accumulators of a power of two of columns each; the epilogue reads 32 columns at a time.
  shape.tmem_columns = 64;
  while (shape.tmem_columns < 2 * shape.tile_rows)
    shape.tmem_columns *= 2;
  static PerDeviceOnce configured;
  if (configured.run([] {
        return cudaFuncSetAttribute(pair_linear_kernel<mode, wide>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    ring_budget + 1024);
      }) != cudaSuccess) {
    return -10;
  }
  const int items = ((plan.tiles - arguments.tail_tiles) * arguments.splits +
                     arguments.tail_tiles * arguments.tail_splits) *
                    shape.row_tiles;
  const int pairs = items < plan.ctas / 2 ? items : plan.ctas / 2;
  return launch_clustered(pair_linear_kernel<mode, wide>, dim3(static_cast<unsigned>(2 * pairs)),
                          dim3(pair_threads), static_cast<size_t>(ring_budget) + 1024, stream, 2,
                          plan.weight_map, plan.input_map, arguments, shape) == cudaSuccess
             ? 0
             : -11;
}

} // namespace

bool schedule_pairs(LinearPlan *plan) {
  LinearPlan &result = *plan;
  // The tail has to begin with a tile of 256 (it does on any even number of SMs).
  if ((result.tiles - result.tail_tiles) % 2 != 0 && result.tail_tiles > 0)
    return false;
  result.tile_width = pair_features;
  result.padded_rows = pair_tile_rows(result.rows, result.element_bytes);
  result.tiles = (result.tiles + 1) / 2;
  result.tail_tiles = (result.tail_tiles + 1) / 2;
  return true;
}

int launch_pair_linear(const LinearPlan &plan, const KernelArguments &arguments, int mode,
                       cudaStream_t stream) {
  const bool wide = plan.element_bytes == 2;
  switch (mode) {
  case 0:
    return wide ? launch_pairs<0, true>(plan, arguments, stream)
                : launch_pairs<0, false>(plan, arguments, stream);
  case 1:
    return wide ? launch_pairs<1, true>(plan, arguments, stream)
                : launch_pairs<1, false>(plan, arguments, stream);
  case 2:
    return wide ? launch_pairs<2, true>(plan, arguments, stream)
                : launch_pairs<2, false>(plan, arguments, stream);
  default:
    return -12;
  }
}

} // namespace carat_b200
