// CTA-pair block-FP8 GEMM (compact FP32 scales) for large M on sm_100a. Same product as
// gemm_block_fp8.cuh, C = cvt(alpha * sum_kb (A[:, kb] B[:, kb]^T) * sfa[m, kb] * sfb[n/128, kb]),
// with the same order of operations for every element.
//
// Two CTAs of a cluster own a 256 x 256 output tile (tcgen05 cta_group::2). Each loads its own 128
// rows of A and half of the B tile's rows, 32 KiB per k-block instead of the 48 KiB of the
// single-CTA kernel, whose 128 x 256 tile alone asks L2 for more than the ~72 B/clk an SM gets.
//
// A k-block is multiplied as two 128-column halves, each into a tensor-memory buffer of its own;
// four buffers fill the 512 columns. A buffer's round trip is MMA -> commit -> promotion -> hand-back
// to the issuer (across the pair), and only what is not MMA of that buffer has to hide behind the
// other buffers: with two 256-column buffers half of the round is MMA time and the hand-over
// latencies (several hundred cycles) show, with four of 128 columns a quarter is.
//
// Warps (20 per CTA): 0 = TMA producer; 1 and 2 = MMA issuers of the two halves (leader; in the peer
// warp 1 relays its full stages); 3 = scales; 4..19 = promotion and epilogue: 128 accumulator rows x
// 64 columns per group of four warps, in FP32 registers. One issuing thread would be the bottleneck:
// the waits, four MMAs and commits of a half take it some 350 cycles, and a half is 256 cycles of
// MMA. The scales of eight k-blocks at a time are multiplied (sfa * sfb) into shared memory by
// warp 3: with every promotion warp loading its own rows' scales each load touched 32 cache lines,
// half of the load unit's time (one issuer and such loads: 561 us at 4096 x 18432 x 7168).
//
// Hand-shakes across the pair: a barrier that the other CTA (or the pair's tensor core) signals is
// waited for with cluster-scope acquire, as in gemm_blockscaled_pair.cuh: the leader's full, empty and
// part_empty, the peer's empty, part_full in both. Between the CTAs only asynchronous copies and
// tensor memory change hands, never ordinary memory: a promotion warp's reads of a buffer have
// completed (tcgen05.wait::ld) and are ordered before its arrival by tcgen05.fence::before_thread_sync,
// the issuer's MMA after its wait by the fence::after_thread_sync. The arrivals therefore keep the
// default scope: with cluster-scope release on part_empty 4096 x 18432 x 7168 takes 950 us, not 487.
//
// Measured (device time back to back, single-CTA kernel -> this one): 4096 x 18432 x 7168 531 -> 493 us
// (2.20 PFLOP/s), 8192 x 4096 x 4096 164 -> 146, 256 x 7168 x 7168 37.0 -> 35.1 (one tile per pair). What is
// left: without the promotion FMAs 4096 x 18432 x 7168 ran in 414 us, without tensor-memory loads too in
// 388, MMAs and operand loads alone took 333, on a box where all of it took 499.
// Slower variants: eight promotion warps of 128 columns (557), 32-column tensor-memory loads (590),
// register re-allocation to 104 for the promotion warps (534). No faster over several runs: packed
// FMA (492-546), three stages (496-558).
#pragma once

#include "gemm_block_fp8.cuh"

namespace b12x_b200 {

struct BlockFp8PairTile {
  static constexpr int BM = 128;                     // rows per CTA (256 per pair)
  static constexpr int BN = 256;
  static constexpr int kHalf = 128;                  // columns of one tensor-memory buffer
  static constexpr int kBuffers = 4;
  static constexpr int kABytes = BM * 128;
  static constexpr int kBHalfBytes = (kHalf / 2) * 128;   // this CTA's rows of one half of B
  static constexpr int kStageBytes = kABytes + 2 * kBHalfBytes;
  static constexpr int kStages = 4;
  static constexpr int kBatch = 8;                         // k-blocks whose scales come together
  static constexpr int kScaleSlots = 3;
  static constexpr int kScalePitch = BM + 4;               // floats between k-blocks (bank spread)
  static constexpr int kScaleFloats = 2 * kBatch * kScalePitch;  // [half][k-block][row]
  static constexpr int kScaleBytes = kScaleSlots * kScaleFloats * 4;
  static constexpr int kCStageBytes = BM * BN * 2;   // four sub-tiles of 128 rows x 64 columns
  static constexpr int kBarrierBytes = 1024;
  static constexpr int kSmemBytes = kStages * kStageBytes + kCStageBytes + kScaleBytes + kBarrierBytes + 1024;
  static constexpr int kFirstPromotionWarp = 4;
  static constexpr int kPromotionWarps = 16;
  static constexpr int kThreads = 32 * (kFirstPromotionWarp + kPromotionWarps);
  static_assert(kSmemBytes <= 227 * 1024, "shared memory overflow");
};

// tiles_m of the parameters counts 256-row pair tiles here. BIAS as in gemm_block_fp8_kernel.
template <bool BIAS>
__global__ void __launch_bounds__(BlockFp8PairTile::kThreads, 1)
gemm_block_fp8_pair_kernel(const __grid_constant__ CUtensorMap map_a,
                           const __grid_constant__ CUtensorMap map_b,
                           const __grid_constant__ CUtensorMap map_c, const BlockFp8Params p) {
  using T = BlockFp8PairTile;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* c_stage = smem + T::kStages * T::kStageBytes;
  float* scales = reinterpret_cast<float*>(c_stage + T::kCStageBytes);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(c_stage + T::kCStageBytes + T::kScaleBytes);
  uint64_t* empty_bar = full_bar + T::kStages;
  uint64_t* part_full_bar = empty_bar + T::kStages;
  uint64_t* part_empty_bar = part_full_bar + T::kBuffers;  // used in the leader only
  uint64_t* scale_full_bar = part_empty_bar + T::kBuffers;
  uint64_t* scale_empty_bar = scale_full_bar + T::kScaleSlots;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(scale_empty_bar + T::kScaleSlots);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  const bool leader = (rank == 0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < T::kStages; ++s) {
      mbar_init(&full_bar[s], leader ? 2 : 1);  // own copies (+ the peer's, relayed)
      mbar_init(&empty_bar[s], leader ? 2 : 1); // one commit per half (peer: the leader's producer)
    }
    for (int b = 0; b < T::kBuffers; ++b) {
      mbar_init(&part_full_bar[b], 1);
      mbar_init(&part_empty_bar[b], T::kPromotionWarps);  // half the warps of each CTA
    }
    for (int s = 0; s < T::kScaleSlots; ++s) {
      mbar_init(&scale_full_bar[s], 1);
      mbar_init(&scale_empty_bar[s], T::kPromotionWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    if (p.use_tma_store) tma_prefetch_desc(&map_c);
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anyone signals across the pair
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const bool tmem_ok = (tmem_base == 0);  // the CTA owns the whole TMEM, so the base is column 0
  if (!tmem_ok && threadIdx.x == 0 && p.status) atomicMax(p.status, kStatusTmemLayout);

  const int num_tiles = p.tiles_m * p.tiles_n;
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int k_blocks = p.k / 128;
  const uint32_t smem_u32 = smem_addr_u32(smem);

  if (!tmem_ok) {
    // fall through to the common tear-down
  } else if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    bool wrapped = false;   // the stages have been used before
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      int tm, tn;
      tile_coords(tile, p.tiles_m, p.tiles_n, p.group_m, tm, tn);
      const int m0 = tm * 256 + static_cast<int>(rank) * T::BM;
      const int n0 = tn * T::BN + static_cast<int>(rank) * (T::kHalf / 2);
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_bounded_cluster(&empty_bar[stage], phase ^ 1, abort_flag)) {
          *abort_flag = 1;
          if (p.status && lane == 0) atomicMax(p.status, kStatusProducerTimeout);
          ok = false;
          break;
        }
        if (elect_one()) {
          // The issuers free a stage in the leader, which passes it on to the peer.
          if (leader && wrapped) mbar_arrive_cluster(map_to_cta(smem_addr_u32(&empty_bar[stage]), 1));
          uint8_t* st = smem + stage * T::kStageBytes;
          mbar_arrive_expect_tx(&full_bar[stage], T::kStageBytes);
          tma_load_2d(st, &map_a, &full_bar[stage], kb * 128, m0);
          tma_load_2d(st + T::kABytes, &map_b, &full_bar[stage], kb * 128, n0);
          tma_load_2d(st + T::kABytes + T::kBHalfBytes, &map_b, &full_bar[stage], kb * 128,
                      n0 + T::kHalf);
        }
        __syncwarp();
        if (++stage == T::kStages) { stage = 0; phase ^= 1; wrapped = true; }
      }
    }
  } else if (warp == 1 && !leader) {
    // ------------------------------ relay (peer CTA) ------------------------------
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      for (int kb = 0; kb < k_blocks; ++kb) {
        if (!mbar_wait_bounded(&full_bar[stage], phase, abort_flag)) {
          *abort_flag = 1;
          if (p.status && lane == 0) atomicMax(p.status, kStatusMmaTimeout);
          ok = false;
          break;
        }
        if (elect_one()) mbar_arrive_cluster(map_to_cta(smem_addr_u32(&full_bar[stage]), 0));
        __syncwarp();
        if (++stage == T::kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1 || warp == 2) {
    // --------------------- MMA issuers, one per half (leader CTA) ---------------------
    const uint32_t half = static_cast<uint32_t>(warp) - 1;
    constexpr uint32_t idesc = make_idesc_f8(256, T::kHalf);
    int stage = 0;
    uint32_t phase = 0;
    uint32_t it = 0;
    bool ok = leader;   // the peer has nothing to issue
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      for (int kb = 0; kb < k_blocks; ++kb, ++it) {
        const uint32_t st = smem_u32 + stage * T::kStageBytes;
        const uint64_t adesc = make_kmajor_sw128_desc(st);
        const uint64_t bdesc = make_kmajor_sw128_desc(st + T::kABytes + half * T::kBHalfBytes);
        const uint32_t buf = (it & 1) * 2 + half;
        if (!mbar_wait_bounded_cluster(&full_bar[stage], phase, abort_flag) ||
            !mbar_wait_bounded_cluster(&part_empty_bar[buf], ((it >> 1) & 1) ^ 1, abort_flag)) {
          *abort_flag = 1;
          if (p.status && lane == 0) atomicMax(p.status, kStatusMmaTimeout);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            tc_mma_f8_pair(buf * T::kHalf, adesc + 2 * j, bdesc + 2 * j, idesc, j > 0 ? 1u : 0u);
          tc_commit_pair_both(smem_addr_u32(&part_full_bar[buf]));
          tc_commit_pair(smem_addr_u32(&empty_bar[stage]));
        }
        __syncwarp();
        if (++stage == T::kStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 3) {
    // ------------------------------ scales (both CTAs) ------------------------------
    uint32_t batch = 0;
    bool ok = true;
    const int n_blocks = p.n / 128;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      int tm, tn;
      tile_coords(tile, p.tiles_m, p.tiles_n, p.group_m, tm, tn);
      const int row0 = (lane >> 3) * 32;   // a lane: one k-block, a quarter of the rows
      const int m0 = tm * 256 + static_cast<int>(rank) * T::BM + row0;
      for (int base = 0; base < k_blocks; base += T::kBatch, ++batch) {
        const uint32_t slot = batch % T::kScaleSlots;
        const int kb = base + (lane & 7);
        const bool live = kb < k_blocks;
        const float w0 = live ? __ldg(p.sfb + static_cast<size_t>(tn * 2) * k_blocks + kb) : 0.0f;
        const float w1 = (live && tn * 2 + 1 < n_blocks)
                             ? __ldg(p.sfb + static_cast<size_t>(tn * 2 + 1) * k_blocks + kb) : 0.0f;
        const float* src = p.sfa + static_cast<size_t>(m0) * k_blocks + kb;
        float x[32];
#pragma unroll
        for (int i = 0; i < 32; ++i)
          x[i] = (live && m0 + i < p.m) ? __ldg(src + static_cast<size_t>(i) * k_blocks) : 0.0f;
        if (!mbar_wait_bounded(&scale_empty_bar[slot], ((batch / T::kScaleSlots) & 1) ^ 1, abort_flag)) {
          *abort_flag = 1;
          if (p.status && lane == 0) atomicMax(p.status, kStatusProducerTimeout);
          ok = false;
          break;
        }
        float* dst = scales + slot * T::kScaleFloats + (lane & 7) * T::kScalePitch + row0;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          *reinterpret_cast<float4*>(dst + i) =
              make_float4(__fmul_rn(x[i], w0), __fmul_rn(x[i + 1], w0), __fmul_rn(x[i + 2], w0),
                          __fmul_rn(x[i + 3], w0));
          *reinterpret_cast<float4*>(dst + T::kBatch * T::kScalePitch + i) =
              make_float4(__fmul_rn(x[i], w1), __fmul_rn(x[i + 1], w1), __fmul_rn(x[i + 2], w1),
                          __fmul_rn(x[i + 3], w1));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&scale_full_bar[slot]);
      }
    }
  } else {
    // ------------------------- promotion + epilogue (both CTAs) -------------------------
    const int quarter = warp & 3;
    const int group = (warp - T::kFirstPromotionWarp) >> 2;  // which 64 of the tile's 256 columns
    const int half = group >> 1;
    constexpr int kCols = 64;
    const float alpha = p.alpha ? *p.alpha : 1.0f;
    uint32_t it = 0;
    uint32_t batch = 0, slot = 0;
    // A warp that gave up a wait keeps walking its tiles (without waiting or storing), because the
    // four warps of a group meet at named barriers.
    bool ok = true;
    bool store_pending = false;
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      int tm, tn;
      tile_coords(tile, p.tiles_m, p.tiles_n, p.group_m, tm, tn);
      const int m0 = tm * 256 + static_cast<int>(rank) * T::BM;
      const int row = m0 + quarter * 32 + lane;
      const int col0 = tn * T::BN + group * kCols;
      float acc[kCols];
#pragma unroll
      for (int i = 0; i < kCols; ++i) acc[i] = 0.0f;
      for (int kb = 0; kb < k_blocks && ok; ++kb, ++it) {
        const uint32_t buf = (it & 1) * 2 + half;
        if ((kb & (T::kBatch - 1)) == 0) {
          slot = batch % T::kScaleSlots;
          ok = mbar_wait_bounded(&scale_full_bar[slot], (batch / T::kScaleSlots) & 1, abort_flag);
          ++batch;
        }
        const float scale = scales[slot * T::kScaleFloats +
                                   (half * T::kBatch + (kb & (T::kBatch - 1))) * T::kScalePitch +
                                   quarter * 32 + lane];
        if (!ok || !mbar_wait_bounded_cluster(&part_full_bar[buf], (it >> 1) & 1, abort_flag)) {
          *abort_flag = 1;
          if (p.status && lane == 0) atomicMax(p.status, kStatusEpilogueTimeout);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t taddr = (static_cast<uint32_t>(quarter * 32) << 16) + buf * T::kHalf +
                               (group & 1) * kCols;
        uint32_t raw[2][16];
        tmem_load_16cols(taddr, raw[0]);
#pragma unroll
        for (int c = 0; c < kCols / 16; ++c) {
          tmem_load_wait();
          if (c + 1 < kCols / 16) {
            tmem_load_16cols(taddr + (c + 1) * 16, raw[(c + 1) & 1]);
          } else {
            // Everything of this buffer is in registers: back to the issuer with it.
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_addr_u32(&part_empty_bar[buf]), 0));
          }
#pragma unroll
          for (int i = 0; i < 16; ++i)
            acc[c * 16 + i] = fmaf(__uint_as_float(raw[c & 1][i]), scale, acc[c * 16 + i]);
        }
        // The slot's last k-block: its scales are in registers.
        if ((kb & (T::kBatch - 1)) == T::kBatch - 1 || kb + 1 == k_blocks) {
          __syncwarp();
          if (lane == 0) mbar_arrive(&scale_empty_bar[slot]);
        }
      }
      if (p.use_tma_store) {
        // The four warps of a group own sub-tile `group`: rows 0..127, 64 columns = 128 bytes
        // per row; 16-byte chunk j of row r sits at position j ^ (r % 8), the layout a
        // 128-byte-swizzled TMA store expects.
        const bool store_thread = (quarter == 0) && (lane == 0);
        if (store_pending) {
          if (store_thread) tma_store_wait_read<0>();
          group_bar_sync(group);
        }
        const int r = quarter * 32 + lane;
        uint8_t* sub = c_stage + group * (128 * 128) + r * 128;
        if constexpr (BIAS) {
          // acc becomes float(cvt(alpha * acc)) + bias; the packing below rounds the sum.
#pragma unroll
          for (int c = 0; c < kCols / 32; ++c) {
            float vals[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) vals[i] = acc[c * 32 + i] * alpha;
            add_bias_32(vals, p.bias, p.out_dtype, col0 + c * 32, p.n);
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[c * 32 + i] = vals[i];
          }
        }
        const float out_scale = BIAS ? 1.0f : alpha;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float lo = acc[j * 8 + 2 * i] * out_scale, hi = acc[j * 8 + 2 * i + 1] * out_scale;
            w[i] = (p.out_dtype == kOutBf16) ? pack_bf16x2(lo, hi) : pack_f16x2(lo, hi);
          }
          *reinterpret_cast<uint4*>(sub + ((j ^ (r & 7)) * 16)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        fence_proxy_async_smem();
        group_bar_sync(group);
        if (store_thread && ok) {
          if (col0 < p.n && m0 < p.m) tma_store_2d(&map_c, c_stage + group * (128 * 128), col0, m0);
          tma_store_commit();
        }
        store_pending = true;
        continue;
      }
      if (!ok) break;
      GemmParams gp;
      gp.c_group_elems = 0;
      gp.c = p.c;
      gp.m = p.m;
      gp.n = p.n;
      gp.ldc = p.ldc;
      gp.out_dtype = p.out_dtype;
#pragma unroll
      for (int c = 0; c < kCols / 32; ++c) {
        float vals[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) vals[i] = acc[c * 32 + i] * alpha;
        if constexpr (BIAS) add_bias_32(vals, p.bias, p.out_dtype, col0 + c * 32, p.n);
        store_row_chunk(gp, 0, row, col0 + c * 32, vals);
      }
    }
    if (p.use_tma_store && quarter == 0 && lane == 0) tma_store_wait_all<0>();
  }

  // Neither CTA leaves while the other may still signal its barriers or read its operands.
  tc_fence_before_sync();
  __syncthreads();
  drain_after_abort(abort_flag);
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace b12x_b200
