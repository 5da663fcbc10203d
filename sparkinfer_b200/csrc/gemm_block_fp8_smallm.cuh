// Weight-streaming block-FP8 GEMM for few activation rows (M <= 128) on sm_100a:
//
//     C[M,N] = cvt(alpha * sum_kb (X[:, kb] W[:, kb]^T) * sfx[m, kb] * sfw[n/128, kb])
//
// Bound: HBM, the weight matrix is read once. The roles of the operands are swapped: 128 weight
// rows are the M side of the tcgen05 MMA, the activation rows (padded to MPAD) its N side. The
// tiled kernel gives such a problem one CTA per 128 x 256 tile: 24 x 7168 x 18432 was 28 CTAs with
// 144 k-blocks in series, 77.9 us.
//
// Split: a cluster of S CTAs owns a weight tile, each CTA streams 1/S of its K; with more tiles
// than SMs S is 1 and the CTAs walk over whole tiles. The FP32 partials of a cluster meet in
// distributed shared memory: each warp sums eight rows x 32 columns over the S CTAs in rank order
// (deterministic) and stores them. Partials through global memory (stream-K with a last-arriver
// reduction) cost a fence, an atomic and loads that queue behind the ~200 KiB of weight requests
// an SM has outstanding: 64 x 1024 x 4608 took 62 us that way, 64 x 47232 x 2560 53 us. Whole
// tiles leave up to a tile's time of imbalance between SMs, of which the memory makes up a part: with
// 16 x 47232 x 7168 on 37, 74, 100, 124 of the SMs the weights come at 2.2, 4.2, 5.1, 6.2 TB/s, so half of
// the SMs still run at two thirds of the full rate.
//
// FP32 scales cannot ride on a block-scaled MMA, so each unit is multiplied unscaled into one of
// four TMEM buffers (MPAD columns each) and the promotion warps add it to FP32 registers with one
// FMA per element: lane = weight row, column = activation row. A weight row block has one scale
// per unit and an activation row another, so the factor of a column is the same for all lanes. A
// warp of its own brings the scales in, eight k-blocks at a time (one 32-byte sector per activation
// row) and up to four such batches ahead, and leaves the products in shared memory as
// [k-block][activation row], where the promotion warps read them as 16-byte broadcasts. (Ordinary
// loads queue behind the ~200 KiB of weight requests an SM has outstanding and take microseconds:
// with the promotion warps loading their own scales 24 x 7168 x 18432 took 31 us.)
//
// Measured (device time back to back, weights from HBM, tiled kernel -> this one): 24 x 7168 x 18432
// 79.5 -> 27.8 us (4.8 TB/s), 1 x 1024 x 4608 24.5 -> 6.1, 64 x 47232 x 2560 34.9 -> 26.9. Of that the wait
// before the weight costs about 1 us, which a stream that began beside the predecessor had saved.
//
// Threads: warp 0 weight producer (and barrier set-up), warp 1 MMA issuer and TMEM owner, warp 2
// activation producer, warp 3 scales, then four promotion warps per 16 or 32 activation rows, which
// keep the sums in registers (with all of 64 rows in one group of four warps, each waits too long
// for its own tensor-memory loads: 64 x 47232 x 2560 33 us instead of 27).
//
// Order on the stream: that of an ordinary launch. The kernel is launched with programmatic stream
// serialization, but every operand, the weight too, is read behind griddepcontrol.wait: an FP32-scaled
// weight is often written by kernels that are not this library's, and one that releases its
// dependents early would otherwise still be writing it. (The block-scaled decode kernel streams its
// weight earlier, on a condition its callers know.) The next grid is released behind the wait as
// well, so that it cannot start beside a grid that this one itself has to wait for.
#pragma once

#include "gemm_blockscaled.cuh"
#include "store_rows.cuh"

namespace b12x_b200 {

template <int MPAD>
struct BlockFp8SmallTile {
  static_assert(MPAD == 16 || MPAD == 32 || MPAD == 64 || MPAD == 128, "padded rows");
  static constexpr int kCols = MPAD <= 32 ? 16 : 32;            // columns of a promotion warp
  static constexpr int kGroups = MPAD / kCols;                  // promotion warp groups of four
  static constexpr int kThreads = 128 + 128 * kGroups;
  static constexpr int kWBytes = 128 * 128;
  static constexpr int kXBytes = MPAD * 128;
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kScalePitch = MPAD + 4;                  // floats between k-blocks (bank spread)
  static constexpr int kBatch = 8;                              // k-blocks whose scales come together
  static constexpr int kScaleSlots = 4;
  static constexpr int kScaleFloats = kBatch * kScalePitch;
  // Barriers, output staging, scales.
  static constexpr int kTailBytes = 1024 + 4 * kGroups * 512 + kScaleSlots * kScaleFloats * 4;
  static constexpr int kStagesRaw = (227 * 1024 - 1024 - kTailBytes) / kStageBytes;
  static constexpr int kStages = kStagesRaw > 12 ? 12 : kStagesRaw;
  static constexpr int kSmemBytes = kStages * kStageBytes + kTailBytes + 1024;
  static constexpr int kBuffers = 4;
  static constexpr int kTmemCols = kBuffers * MPAD;             // 64, 128, 256 or 512
};

struct BlockFp8SmallParams {
  const float* sfx;    // [M, K/128]
  const float* sfw;    // [N/128, K/128]
  void* c;
  const float* alpha;
  const void* bias;    // [N] values of the output dtype added to every row, or null
  int* status;
  int m, n, ldc, out_dtype;
  int tiles, k_blocks;
  int split;             // CTAs of a cluster = CTAs per tile
  int packed_store;      // 2-byte outputs with 16-byte aligned rows
};

// Eight output rows x 32 columns of a warp (lane = column): scale, bias, round, store.
__device__ __forceinline__ void store_block_fp8_rows8(const BlockFp8SmallParams& p, uint8_t* staging,
                                                      int lane, float alpha, int row0, int col0,
                                                      float (&vals)[8]) {
  const int col = col0 + lane;
  const float bias = p.bias != nullptr ? load_bias_1(p.bias, p.out_dtype, col, p.n) : 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    vals[i] *= alpha;
    if (p.bias != nullptr) vals[i] = add_bias_1(vals[i], bias, p.out_dtype);
  }
  if (p.packed_store) {
    store_rows8_packed(p, reinterpret_cast<uint16_t*>(staging), lane, 0, row0, col0, vals);
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (row0 + i >= p.m || col >= p.n) continue;
    const size_t idx = static_cast<size_t>(row0 + i) * p.ldc + col;
    if (p.out_dtype == kOutBf16)
      static_cast<__nv_bfloat16*>(p.c)[idx] = __float2bfloat16_rn(vals[i]);
    else if (p.out_dtype == kOutFp16)
      static_cast<__half*>(p.c)[idx] = __float2half_rn(vals[i]);
    else
      static_cast<float*>(p.c)[idx] = vals[i];
  }
}

__device__ __forceinline__ float ld_shared_cluster_f32(uint32_t cluster_addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
  return v;
}

template <int MPAD>
__global__ void __launch_bounds__(BlockFp8SmallTile<MPAD>::kThreads, 1)
gemm_block_fp8_smallm_kernel(const __grid_constant__ CUtensorMap map_w,
                             const __grid_constant__ CUtensorMap map_x,
                             const BlockFp8SmallParams p) {
  using T = BlockFp8SmallTile<MPAD>;
  constexpr int CW = T::kCols;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + T::kStages * T::kStageBytes);
  uint64_t* empty_bar = full_bar + T::kStages;
  uint64_t* part_full_bar = empty_bar + T::kStages;
  uint64_t* part_empty_bar = part_full_bar + T::kBuffers;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(part_empty_bar + T::kBuffers);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* scale_full_bar = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(full_bar) + 512);
  uint64_t* scale_empty_bar = scale_full_bar + T::kScaleSlots;
  float* scales = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(full_bar) + 1024 +
                                           4 * T::kGroups * 512);
  uint8_t* staging = reinterpret_cast<uint8_t*>(full_bar) + 1024;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // This CTA: k-blocks [kb_begin, kb_end) of tiles tile0, tile0 + tile_step, ... (one tile when
  // it is split).
  const int rank = static_cast<int>(blockIdx.x) % p.split;
  const int tile0 = static_cast<int>(blockIdx.x) / p.split;
  const int tile_step = static_cast<int>(gridDim.x) / p.split;
  const int kb_begin = static_cast<int>(static_cast<long long>(p.k_blocks) * rank / p.split);
  const int kb_end = static_cast<int>(static_cast<long long>(p.k_blocks) * (rank + 1) / p.split);

  if (warp == 0) {
    // ------------------------------ weight producer ------------------------------
    if (lane == 0) {
      *abort_flag = 0;
      for (int s = 0; s < T::kStages; ++s) {
        mbar_init(&full_bar[s], 2);  // weight producer + activation producer
        mbar_init(&empty_bar[s], 1);
      }
      for (int b = 0; b < T::kBuffers; ++b) {
        mbar_init(&part_full_bar[b], 1);
        mbar_init(&part_empty_bar[b], 4 * T::kGroups);
      }
      for (int b = 0; b < T::kScaleSlots; ++b) {
        mbar_init(&scale_full_bar[b], 1);
        mbar_init(&scale_empty_bar[b], 4 * T::kGroups);
      }
      fence_mbar_init();
      fence_proxy_async_smem();
      tma_prefetch_desc(&map_w);
    }
    __syncwarp();
    asm volatile("barrier.cta.arrive 3, %0;" ::"n"(T::kThreads) : "memory");
    grid_dependency_wait();    // the weight may come from the previous grid
    grid_launch_dependents();  // every CTA of which has finished by now
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = tile0; tile < p.tiles && ok; tile += tile_step) {
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        if (!mbar_wait_bounded(&empty_bar[stage], phase ^ 1, abort_flag)) {
          *abort_flag = 1;
          if (p.status && lane == 0) atomicMax(p.status, kStatusProducerTimeout);
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_arrive_expect_tx(&full_bar[stage], T::kWBytes);
          tma_load_2d(smem + stage * T::kStageBytes, &map_w, &full_bar[stage], kb * 128, tile * 128);
        }
        __syncwarp();
        if (++stage == T::kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else {
    if (warp == 1) tmem_alloc(tmem_slot, T::kTmemCols);
    tc_fence_before_sync();
    asm volatile("barrier.cta.sync 3, %0;" ::"n"(T::kThreads) : "memory");
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const bool tmem_ok = (tmem_base >> 16) == 0;
    if (!tmem_ok && threadIdx.x == 32) {
      *abort_flag = 1;
      if (p.status) atomicMax(p.status, kStatusTmemLayout);
    }
    if (!tmem_ok) {
      // nothing is issued; everyone leaves through the common tear-down
    } else if (warp == 2) {
      // ------------------------------ activation producer ------------------------------
      if (lane == 0) tma_prefetch_desc(&map_x);
      grid_dependency_wait();  // activations may come from the previous grid
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = tile0; tile < p.tiles && ok; tile += tile_step) {
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!mbar_wait_bounded(&empty_bar[stage], phase ^ 1, abort_flag)) {
            *abort_flag = 1;
            if (p.status && lane == 0) atomicMax(p.status, kStatusProducerTimeout);
            ok = false;
            break;
          }
          if (elect_one()) {
            mbar_arrive_expect_tx(&full_bar[stage], T::kXBytes);
            tma_load_2d(smem + stage * T::kStageBytes + T::kWBytes, &map_x, &full_bar[stage], kb * 128, 0);
          }
          __syncwarp();
          if (++stage == T::kStages) { stage = 0; phase ^= 1; }
        }
      }
    } else if (warp == 1) {
      // ------------------------------ MMA issuer ------------------------------
      constexpr uint32_t idesc = make_idesc_f8(128, MPAD);
      const uint32_t smem_u32 = smem_addr_u32(smem);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t it = 0;
      bool ok = true;
      for (int tile = tile0; tile < p.tiles && ok; tile += tile_step) {
        for (int kb = kb_begin; kb < kb_end; ++kb, ++it) {
          const uint32_t buf = it % T::kBuffers;
          if (!mbar_wait_bounded(&full_bar[stage], phase, abort_flag) ||
              !mbar_wait_bounded(&part_empty_bar[buf], ((it / T::kBuffers) & 1) ^ 1, abort_flag)) {
            *abort_flag = 1;
            if (p.status && lane == 0) atomicMax(p.status, kStatusMmaTimeout);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          if (elect_one()) {
            const uint32_t st = smem_u32 + stage * T::kStageBytes;
            const uint64_t wdesc = make_kmajor_sw128_desc(st);
            const uint64_t xdesc = make_kmajor_sw128_desc(st + T::kWBytes);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              tc_mma_f8(tmem_base + buf * MPAD, wdesc + 2 * j, xdesc + 2 * j, idesc, j > 0 ? 1u : 0u);
            tc_commit(&empty_bar[stage]);
            tc_commit(&part_full_bar[buf]);
          }
          __syncwarp();
          if (++stage == T::kStages) { stage = 0; phase ^= 1; }
        }
      }
    } else if (warp == 3) {
      // ------------------------------ scales ------------------------------
      grid_dependency_wait();  // activation scales may come from the previous grid
      uint32_t batch = 0;
      bool ok = true;
      for (int tile = tile0; tile < p.tiles && ok; tile += tile_step) {
        for (int base = kb_begin; base < kb_end && ok; base += T::kBatch, ++batch) {
          const uint32_t slot = batch % T::kScaleSlots;
          constexpr int kRows = MPAD / 4;   // a lane: one k-block, a quarter of the rows
          const int row0 = (lane >> 3) * kRows;
          const int kb = base + (lane & 7);
          const bool live = kb < kb_end;
          const float w = live ? ld_global_f32(p.sfw + static_cast<size_t>(tile) * p.k_blocks + kb) : 0.0f;
          const float* src = p.sfx + static_cast<size_t>(row0) * p.k_blocks + kb;
          float x[kRows];
#pragma unroll
          for (int i = 0; i < kRows; ++i)
            x[i] = (live && row0 + i < p.m) ? ld_global_f32(src + static_cast<size_t>(i) * p.k_blocks) : 0.0f;
          if (!mbar_wait_bounded(&scale_empty_bar[slot], ((batch / T::kScaleSlots) & 1) ^ 1, abort_flag)) {
            *abort_flag = 1;
            if (p.status && lane == 0) atomicMax(p.status, kStatusProducerTimeout);
            ok = false;
            break;
          }
          float* dst = scales + slot * T::kScaleFloats + (lane & 7) * T::kScalePitch + row0;
#pragma unroll
          for (int i = 0; i < kRows; i += 4)
            *reinterpret_cast<float4*>(dst + i) =
                make_float4(__fmul_rn(x[i], w), __fmul_rn(x[i + 1], w), __fmul_rn(x[i + 2], w),
                            __fmul_rn(x[i + 3], w));
          __syncwarp();
          if (lane == 0) mbar_arrive(&scale_full_bar[slot]);
        }
      }
    } else if (warp >= 4) {
      // ------------------------- promotion and output -------------------------
      grid_dependency_wait();  // alpha and C
      const int quarter = warp & 3;
      const int m0 = ((warp - 4) >> 2) * CW;      // first activation row of this warp
      const int n_local = quarter * 32 + lane;    // weight row inside the tile
      const float alpha = p.alpha ? *p.alpha : 1.0f;
      uint32_t it = 0, batch = 0;
      bool ok = true;
      for (int tile = tile0; tile < p.tiles && ok; tile += tile_step) {
        float acc[CW];
#pragma unroll
        for (int i = 0; i < CW; ++i) acc[i] = 0.0f;
        for (int base = kb_begin; base < kb_end && ok; base += T::kBatch, ++batch) {
          const uint32_t slot = batch % T::kScaleSlots;
          const float* scale = scales + slot * T::kScaleFloats + m0;
          const int count = min(T::kBatch, kb_end - base);
          for (int j = 0; j < count; ++j, ++it, scale += T::kScalePitch) {
            const uint32_t buf = it % T::kBuffers;
            if ((j == 0 && !mbar_wait_bounded(&scale_full_bar[slot], (batch / T::kScaleSlots) & 1, abort_flag)) ||
                !mbar_wait_bounded(&part_full_bar[buf], (it / T::kBuffers) & 1, abort_flag)) {
              *abort_flag = 1;
              if (p.status && lane == 0) atomicMax(p.status, kStatusEpilogueTimeout);
              ok = false;
              break;
            }
            tc_fence_after_sync();
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * MPAD + m0;
            uint32_t raw[CW / 16][16];
#pragma unroll
            for (int c = 0; c < CW / 16; ++c) tmem_load_16cols(taddr + c * 16, raw[c]);
            tmem_load_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&part_empty_bar[buf]);
#pragma unroll
            for (int i = 0; i < CW; i += 4) {
              const float4 f = *reinterpret_cast<const float4*>(scale + i);
              acc[i] = fmaf(__uint_as_float(raw[i / 16][i % 16]), f.x, acc[i]);
              acc[i + 1] = fmaf(__uint_as_float(raw[i / 16][i % 16 + 1]), f.y, acc[i + 1]);
              acc[i + 2] = fmaf(__uint_as_float(raw[i / 16][i % 16 + 2]), f.z, acc[i + 2]);
              acc[i + 3] = fmaf(__uint_as_float(raw[i / 16][i % 16 + 3]), f.w, acc[i + 3]);
            }
          }
          __syncwarp();
          if (ok && lane == 0) mbar_arrive(&scale_empty_bar[slot]);
        }
        if (p.split > 1) {
          // Every load of this CTA has been consumed (its last MMA is in `acc`), so the ring can
          // hold the partial: [row][128 columns].
          float* part = reinterpret_cast<float*>(smem);
#pragma unroll
          for (int i = 0; i < CW; ++i) part[(m0 + i) * 128 + n_local] = acc[i];
        } else if (ok) {
#pragma unroll
          for (int r0 = 0; r0 < CW; r0 += 8) {
            if (m0 + r0 >= p.m) break;
            float vals[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) vals[i] = acc[r0 + i];
            store_block_fp8_rows8(p, staging + (warp - 4) * 512, lane, alpha, m0 + r0,
                                  tile * 128 + quarter * 32, vals);
          }
        }
      }
    }
  }

  if (p.split > 1) {
    // Uniform over the cluster: every thread of every CTA meets here twice, also after a timeout.
    __syncwarp();
    cluster_sync_all();
    if (warp >= 4 && *abort_flag == 0) {
      const float alpha = p.alpha ? *p.alpha : 1.0f;
      constexpr int kWarps = 4 * T::kGroups;
      const uint32_t part = smem_addr_u32(smem);
      const int row_groups = (p.m + 7) / 8;
      for (int item = rank + p.split * (warp - 4); item < row_groups * 4; item += p.split * kWarps) {
        const int r0 = (item >> 2) * 8, col0 = (item & 3) * 32;
        float sum[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) sum[i] = 0.0f;
        // Two CTAs' values in flight at a time; added in rank order.
        for (int s = 0; s < p.split; s += 2) {
          float v[2][8];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t src = map_to_cta(part, min(s + h, p.split - 1)) + (r0 * 128 + col0 + lane) * 4;
#pragma unroll
            for (int i = 0; i < 8; ++i) v[h][i] = ld_shared_cluster_f32(src + i * 512);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (s + h < p.split) {
#pragma unroll
              for (int i = 0; i < 8; ++i) sum[i] += v[h][i];
            }
        }
        store_block_fp8_rows8(p, staging + (warp - 4) * 512, lane, alpha, r0, tile0 * 128 + col0, sum);
      }
    }
    __syncwarp();
    cluster_sync_all();  // nobody leaves while its partial is being read
  }

  tc_fence_before_sync();
  __syncthreads();
  drain_after_abort(abort_flag);
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(*tmem_slot, T::kTmemCols);
  }
}

}  // namespace b12x_b200
