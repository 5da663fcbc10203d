// Host side of the block-FP8 GEMM (E4M3 operands with FP32 scales): argument checks, kernel choice,
// launches.
#include "host_common.cuh"

#include "gemm_block_fp8.cuh"
#include "gemm_block_fp8_pair.cuh"
#include "gemm_block_fp8_smallm.cuh"

using namespace b12x_b200;

namespace {

// ------------------------------------------------------------------------------------------
// Weight-streaming kernel: few activation rows
// ------------------------------------------------------------------------------------------
// Largest M of the weight-streaming kernel. Up to 64 rows it is never behind the tiled kernel
// (device time, weights from HBM: 64 x 54528 x 768 13.0 against 16.4 us, 64 x 7168 x 18432 31 against
// 81). From 65 to 128 rows its activation traffic doubles, and it is ahead only where the tiled
// kernel leaves SMs idle: 128 x 7168 x 18432 43 against 82 us, 128 x 1024 x 4608 11 against 26, but
// 128 x 47232 x 2560 (185 tiles of 256 columns) 38 against 34.
constexpr int64_t kBlockFp8SmallM = 128;
constexpr int64_t kBlockFp8SmallMAlways = 64;

// Clusters of `size` CTAs with an SM each that the current device can hold at once: a cluster
// lives inside one GPC, so SMs left over in a GPC stay idle (148 SMs hold 74, 48, 33, 26, 22, 15
// and 15 clusters of 2 to 8). Asked once per device and size.
int max_clusters(int size) {
  static std::atomic<int> cache[64][9];  // 0: not asked yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || size < 1 || size > 8) return 0;
  int have = cache[dev][size];
  if (have != 0) return have - 1;
  using T = BlockFp8SmallTile<16>;
  cudaFuncSetAttribute(gemm_block_fp8_smallm_kernel<16>,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmemBytes);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(unsigned(size), 1, 1);
  cfg.blockDim = dim3(T::kThreads, 1, 1);
  cfg.dynamicSmemBytes = T::kSmemBytes;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(size);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int count = 0;
  if (cudaOccupancyMaxActiveClusters(&count, gemm_block_fp8_smallm_kernel<16>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    count = 0;
  }
  cache[dev][size] = count + 1;
  return count;
}

struct BlockFp8SmallPlan {
  int m_pad, tiles, k_blocks, split, grid;
};

// False when the shape does not belong to the kernel.
bool plan_block_fp8_small(int64_t m, int64_t n, int64_t k, int sms, BlockFp8SmallPlan* pl) {
  if (m < 1 || m > kBlockFp8SmallM) return false;
  if (m > kBlockFp8SmallMAlways && (n + BlockFp8Tile::BN - 1) / BlockFp8Tile::BN > sms / 2) return false;
  pl->m_pad = m <= 16 ? 16 : m <= 32 ? 32 : m <= 64 ? 64 : 128;
  const int64_t tiles = n / 128, k_blocks = k / 128;
  pl->tiles = int(tiles);
  pl->k_blocks = int(k_blocks);
  // As many CTAs per tile as the SMs allow, at most a portable cluster of eight and no more than
  // the tile has k-blocks, and all clusters resident at once (17 clusters of eight ran in two
  // rounds: 1 x 2176 x 7168 11.3 us, 7.3 with clusters of six); more tiles than SMs are walked
  // over whole.
  int64_t split = sms / tiles;
  if (split > 8) split = 8;
  if (split > k_blocks) split = k_blocks;
  if (split < 1) split = 1;
  while (split > 1 && tiles > max_clusters(int(split))) --split;
  pl->split = int(split);
  pl->grid = int(split > 1 ? tiles * split : (tiles < sms ? tiles : sms));
  return true;
}

template <int MPAD>
int launch_block_fp8_small(const void* a, const void* b, const BlockFp8SmallParams& p, int64_t k,
                           int grid, cudaStream_t stream) {
  using T = BlockFp8SmallTile<MPAD>;
  CUtensorMap map_w, map_x;
  int rc = make_operand_map_2d(&map_w, b, uint64_t(p.n), uint64_t(k), 128);
  if (rc != B12X_B200_OK) return rc;
  rc = make_operand_map_2d(&map_x, a, uint64_t(p.m), uint64_t(k), MPAD);
  if (rc != B12X_B200_OK) return rc;
  static std::atomic<bool> set_for[64];  // zero-initialised; setting the attribute twice is harmless
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !set_for[dev]) {
    const cudaError_t err =
        cudaFuncSetAttribute(gemm_block_fp8_smallm_kernel<MPAD>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmemBytes);
    if (err != cudaSuccess) return fail_cuda(err, "cudaFuncSetAttribute");
    set_for[dev] = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(unsigned(grid), 1, 1);
  cfg.blockDim = dim3(T::kThreads, 1, 1);
  cfg.dynamicSmemBytes = T::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(p.split);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = switches().decode_overlap ? 2 : 1;
  const cudaError_t err =
      cudaLaunchKernelEx(&cfg, gemm_block_fp8_smallm_kernel<MPAD>, map_w, map_x, p);
  if (err != cudaSuccess) return fail_cuda(err, "gemm_block_fp8_smallm launch");
  return B12X_B200_OK;
}

int run_block_fp8_small(const BlockFp8SmallPlan& pl, const void* a, const float* sfa, const void* b,
                        const float* sfb, void* c, int c_dtype, const float* alpha, int64_t m,
                        int64_t n, int64_t k, int64_t ldc, const void* bias,
                        int* status, cudaStream_t stream) {
  BlockFp8SmallParams p;
  memset(&p, 0, sizeof(p));
  p.sfx = sfa;
  p.sfw = sfb;
  p.c = c;
  p.alpha = alpha;
  p.bias = bias;
  p.status = status;
  p.m = int(m);
  p.n = int(n);
  p.ldc = int(ldc);
  p.out_dtype = c_dtype;
  p.tiles = pl.tiles;
  p.k_blocks = pl.k_blocks;
  p.split = pl.split;
  p.packed_store = (c_dtype != B12X_B200_FP32 && aligned16(c) && ldc % 8 == 0) ? 1 : 0;
  switch (pl.m_pad) {
    case 16: return launch_block_fp8_small<16>(a, b, p, k, pl.grid, stream);
    case 32: return launch_block_fp8_small<32>(a, b, p, k, pl.grid, stream);
    case 64: return launch_block_fp8_small<64>(a, b, p, k, pl.grid, stream);
    default: return launch_block_fp8_small<128>(a, b, p, k, pl.grid, stream);
  }
}

// ------------------------------------------------------------------------------------------
// Tiled kernels
// ------------------------------------------------------------------------------------------
template <bool BIAS>
int launch_block_fp8_pair(const CUtensorMap& map_a, const CUtensorMap& map_b,
                          const CUtensorMap& map_c, const BlockFp8Params& p, int pairs,
                          cudaStream_t stream) {
  using T = BlockFp8PairTile;
  static std::atomic<bool> set_for[64];  // zero-initialised; setting the attribute twice is harmless
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !set_for[dev]) {
    const cudaError_t err =
        cudaFuncSetAttribute(gemm_block_fp8_pair_kernel<BIAS>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmemBytes);
    if (err != cudaSuccess) return fail_cuda(err, "cudaFuncSetAttribute");
    set_for[dev] = true;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(unsigned(2 * pairs), 1, 1);
  cfg.blockDim = dim3(T::kThreads, 1, 1);
  cfg.dynamicSmemBytes = T::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t err =
      cudaLaunchKernelEx(&cfg, gemm_block_fp8_pair_kernel<BIAS>, map_a, map_b, map_c, p);
  if (err != cudaSuccess) return fail_cuda(err, "gemm_block_fp8_pair launch");
  return B12X_B200_OK;
}

// The CTA-pair kernel is faster per round of tiles but has more to do between two tiles. Single-CTA
// against pair kernel in us: K = 512 100 / 109 (8192 x 16384) and 10.3 / 12.5 (1024 x 4096), K = 1536
// 14.5 / 16.6 (700 x 5120), K = 2048 16.6 / 17.4 (200 x 14336) but 138 / 132 (8192 x 7168), K = 3072 18.6 / 18.8
// (160 x 2048), 20.5 / 20.6 (512 x 7168) but 60 / 58 (2048 x 7168), K = 4096 164 / 146 (8192 x 4096), K = 7168
// 37.0 / 35.1 (256 x 7168) and 531 / 493 (4096 x 18432), K = 16384 78 / 72 (2048 x 2048): the line is drawn
// at K = 3072, where one tile per pair is a tie and more are ahead. An odd number of 128-row tiles costs it a row of
// tiles, so it must not need more rounds (640 x 7168: 84 pair tiles are two rounds of 74 pairs,
// 140 single tiles are one of 148 SMs).
bool block_fp8_pair_wins(int64_t m, int64_t n, int64_t k, int sms) {
  if (m <= 128 || k < 3072 || sms < 2) return false;
  const int64_t tiles_n = (n + 255) / 256, pairs = sms / 2;
  const int64_t pair_rounds = ((m + 255) / 256 * tiles_n + pairs - 1) / pairs;
  const int64_t single_rounds = ((m + 127) / 128 * tiles_n + sms - 1) / sms;
  return pair_rounds <= single_rounds;
}

int gemm_block_fp8_impl(const void* a, const float* sfa, const void* b, const float* sfb, void* c,
                        int c_dtype, const float* alpha, int64_t m, int64_t n, int64_t k,
                        int64_t ldc, int sm_count, const b12x_b200_epilogue_t* epilogue,
                        int* status, b12x_b200_stream_t stream) {
  if (c_dtype < B12X_B200_BF16 || c_dtype > B12X_B200_FP32)
    return fail(B12X_B200_ERR_INVALID_ARGUMENT, "unknown output dtype");
  if (m < 0 || n < 0 || k <= 0 || m > INT32_MAX || n > INT32_MAX || k > INT32_MAX)
    return fail(B12X_B200_ERR_INVALID_ARGUMENT, "bad problem size");
  if (n % 128 != 0 || k % 128 != 0)
    return fail(B12X_B200_ERR_UNSUPPORTED, "block-FP8 GEMM needs N and K divisible by 128");
  if (m == 0 || n == 0) return B12X_B200_OK;
  if (!a || !b || !sfa || !sfb || !c) return fail(B12X_B200_ERR_INVALID_ARGUMENT, "null pointer");
  if (ldc < n) return fail(B12X_B200_ERR_INVALID_ARGUMENT, "ldc < n");
  if (!aligned16(a) || !aligned16(b) || (reinterpret_cast<uintptr_t>(sfa) & 3) ||
      (reinterpret_cast<uintptr_t>(sfb) & 3))
    return fail(B12X_B200_ERR_ALIGNMENT, "operands must be 16-byte and scales 4-byte aligned");
  {
    const int erc = check_epilogue(epilogue, c_dtype, n, false);
    if (erc != B12X_B200_OK) return erc;
  }
  DeviceInfo info;
  int rc = device_info(&info);
  if (rc != B12X_B200_OK) return rc;
  if (info.cc_major != 10) return fail(B12X_B200_ERR_NO_DEVICE_CODE, "device is not sm_100");
  const int sms = (sm_count > 0 && sm_count < info.sm_count) ? sm_count : info.sm_count;

  BlockFp8SmallPlan small;
  if (plan_block_fp8_small(m, n, k, sms, &small))
    return run_block_fp8_small(small, a, sfa, b, sfb, c, c_dtype, alpha, m, n, k, ldc,
                               epilogue ? epilogue->bias : nullptr, status,
                               reinterpret_cast<cudaStream_t>(stream));

  const int64_t pair_tiles = ((m + 255) / 256) * ((n + 255) / 256);
  const bool use_pair = block_fp8_pair_wins(m, n, k, sms);

  CUtensorMap map_a, map_b;
  rc = make_operand_map_2d(&map_a, a, uint64_t(m), uint64_t(k), BlockFp8Tile::BM);
  if (rc != B12X_B200_OK) return rc;
  rc = make_operand_map_2d(&map_b, b, uint64_t(n), uint64_t(k),
                           use_pair ? BlockFp8PairTile::kHalf / 2 : BlockFp8Tile::BN);
  if (rc != B12X_B200_OK) return rc;

  BlockFp8Params p;
  p.sfa = sfa;
  p.sfb = sfb;
  p.c = c;
  p.alpha = alpha;
  p.status = status;
  p.m = int(m);
  p.n = int(n);
  p.k = int(k);
  p.ldc = int(ldc);
  p.out_dtype = c_dtype;
  p.tiles_m = int((m + BlockFp8Tile::BM - 1) / BlockFp8Tile::BM);
  p.tiles_n = int((n + BlockFp8Tile::BN - 1) / BlockFp8Tile::BN);
  // Tile rows per group of the tile order: 4096 x 18432 x 7168 warm: 4 -> 525, 8 -> 508,
  // 16 -> 499, 32 (all rows of this problem) -> 496 us.
  p.group_m = 32;
  p.bias = epilogue ? epilogue->bias : nullptr;
  const int64_t tiles = int64_t(p.tiles_m) * p.tiles_n;
  const int grid = int(tiles < sms ? tiles : sms);
  static std::atomic<bool> set_for[64];  // zero-initialised; setting the attribute twice is harmless
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !set_for[dev]) {
    cudaError_t attr_err =
        cudaFuncSetAttribute(gemm_block_fp8_kernel<false>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, BlockFp8Tile::kSmemBytes);
    if (attr_err == cudaSuccess)
      attr_err = cudaFuncSetAttribute(gemm_block_fp8_kernel<true>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      BlockFp8Tile::kSmemBytes);
    if (attr_err != cudaSuccess) return fail_cuda(attr_err, "cudaFuncSetAttribute");
    set_for[dev] = true;
  }
  // Output through TMA when rows of C are 16-byte aligned 2-byte values; otherwise the
  // epilogue stores straight from registers.
  CUtensorMap map_c;
  memset(&map_c, 0, sizeof(map_c));
  p.use_tma_store = 0;
  if (c_dtype != B12X_B200_FP32 && aligned16(c) && (ldc * 2) % 16 == 0) {
    rc = make_output_map_2d(&map_c, c, uint64_t(m), uint64_t(n), uint64_t(ldc));
    if (rc != B12X_B200_OK) return rc;
    p.use_tma_store = 1;
  }
  if (use_pair) {
    p.tiles_m = int((m + 255) / 256);
    p.group_m = 16;
    const int pairs = int(pair_tiles < sms / 2 ? pair_tiles : sms / 2);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    return p.bias ? launch_block_fp8_pair<true>(map_a, map_b, map_c, p, pairs, s)
                  : launch_block_fp8_pair<false>(map_a, map_b, map_c, p, pairs, s);
  }
  if (p.bias)
    gemm_block_fp8_kernel<true><<<grid, BlockFp8Tile::kThreads, BlockFp8Tile::kSmemBytes,
                                  reinterpret_cast<cudaStream_t>(stream)>>>(map_a, map_b, map_c, p);
  else
    gemm_block_fp8_kernel<false><<<grid, BlockFp8Tile::kThreads, BlockFp8Tile::kSmemBytes,
                                   reinterpret_cast<cudaStream_t>(stream)>>>(map_a, map_b, map_c, p);
  const cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return fail_cuda(err, "gemm_block_fp8 launch");
  return B12X_B200_OK;
}

}  // namespace

extern "C" int b12x_b200_gemm_block_fp8(const void* a, const float* sfa, const void* b,
                                        const float* sfb, void* c, int c_dtype,
                                        const float* alpha, int64_t m, int64_t n, int64_t k,
                                        int64_t ldc, int sm_count, int* status,
                                        b12x_b200_stream_t stream) {
  return gemm_block_fp8_impl(a, sfa, b, sfb, c, c_dtype, alpha, m, n, k, ldc, sm_count, nullptr,
                             status, stream);
}

extern "C" int b12x_b200_gemm_block_fp8_ex(const void* a, const float* sfa, const void* b,
                                           const float* sfb, void* c, int c_dtype,
                                           const float* alpha, int64_t m, int64_t n, int64_t k,
                                           int64_t ldc, int sm_count,
                                           const b12x_b200_epilogue_t* epilogue, int* status,
                                           b12x_b200_stream_t stream) {
  return gemm_block_fp8_impl(a, sfa, b, sfb, c, c_dtype, alpha, m, n, k, ldc, sm_count, epilogue,
                             status, stream);
}
