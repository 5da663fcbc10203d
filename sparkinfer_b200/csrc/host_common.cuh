// Host helpers shared by the translation units behind the C ABI: error text, TMA descriptor
// encoding, device properties, switches and the workspace layout.
#pragma once

#include "../../include/b12x_b200.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace b12x_b200 {

// Text of the calling thread's last failure (defined in capi.cu).
extern thread_local char g_last_error[256];

inline int fail_cuda(cudaError_t err, const char* what) {
  snprintf(g_last_error, sizeof(g_last_error), "%s: %s", what, cudaGetErrorString(err));
  return B12X_B200_ERR_CUDA;
}

inline int fail(int code, const char* what) {
  snprintf(g_last_error, sizeof(g_last_error), "%s", what);
  return code;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver entry point is looked up through the runtime so the library carries no link-time
// dependency on libcuda (it must load on machines without a driver).
inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  });
  return fn;
}

// Checks of the optional epilogue description that do not depend on the kernel. `allow_quant`:
// whether the kernel that will run can re-quantize its output (only the decode kernel can).
inline int check_epilogue(const b12x_b200_epilogue_t* e, int c_dtype, int64_t n, bool allow_quant) {
  if (!e) return B12X_B200_OK;
  if (e->bias) {
    const uintptr_t align = (c_dtype == B12X_B200_FP32) ? 3 : 1;
    if (reinterpret_cast<uintptr_t>(e->bias) & align)
      return fail(B12X_B200_ERR_ALIGNMENT, "bias must be aligned to its element size");
  }
  if (e->quant_values) {
    if (!allow_quant)
      return fail(B12X_B200_ERR_UNSUPPORTED,
                  "output re-quantization is available in the decode kernel only (M <= 128)");
    if (c_dtype == B12X_B200_FP32)
      return fail(B12X_B200_ERR_UNSUPPORTED, "output re-quantization needs a BF16 or FP16 output");
    if (n % 32 != 0 || e->quant_cols % 32 != 0 || e->quant_col0 % 32 != 0 || e->quant_col0 < 0 ||
        e->quant_col0 + n > e->quant_cols || e->quant_ld < e->quant_cols ||
        e->quant_cols > INT32_MAX)
      return fail(B12X_B200_ERR_INVALID_ARGUMENT,
                  "re-quantized output: N, quant_col0 and quant_cols must be multiples of 32, "
                  "quant_col0 + N <= quant_cols <= quant_ld");
  } else if (e->quant_scale_rows || e->quant_scale_mma) {
    return fail(B12X_B200_ERR_INVALID_ARGUMENT, "quant scales given without quant_values");
  }
  return B12X_B200_OK;
}

// K-major byte matrix [rows, row_bytes] -> boxes of 128 bytes x box_rows, 128-byte swizzle.
inline int make_operand_map_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes,
                        uint32_t box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(B12X_B200_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t dims[2] = {row_bytes, rows};
  const cuuint64_t strides[1] = {row_bytes};
  const cuuint32_t box[2] = {128, box_rows};
  const cuuint32_t elem_strides[2] = {1, 1};
  const CUresult r =
      fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box,
         elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_last_error, sizeof(g_last_error), "cuTensorMapEncodeTiled failed (%d)", int(r));
    return B12X_B200_ERR_CUDA;
  }
  return B12X_B200_OK;
}

// Stack of `groups` K-major byte matrices [groups, rows, row_bytes] -> boxes of 128 bytes x
// box_rows x 1 group, 128-byte swizzle. A box never crosses into the next group: rows at or
// beyond `rows` are out of bounds and read as zeros. `pitch`: bytes between rows (0: row_bytes),
// for one group only; bytes of a row at or beyond row_bytes read as zeros too.
inline int make_operand_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes,
                     uint32_t box_rows, uint64_t groups = 1, uint64_t pitch = 0) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(B12X_B200_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t dims[3] = {row_bytes, rows, groups};
  if (pitch == 0) pitch = row_bytes;
  const cuuint64_t strides[2] = {pitch, rows * pitch};
  const cuuint32_t box[3] = {128, box_rows, 1};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  const CUresult r =
      fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box,
         elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_last_error, sizeof(g_last_error), "cuTensorMapEncodeTiled failed (%d)", int(r));
    return B12X_B200_ERR_CUDA;
  }
  return B12X_B200_OK;
}

// Row-major BF16 matrix [rows, cols] with row pitch `ld` elements -> unswizzled boxes of
// box_cols x box_rows elements (the raw activation rows of the fused-quantizer decode GEMM).
inline int make_raw_rows_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                      uint32_t box_cols, uint32_t box_rows, uint64_t groups = 1,
                      uint64_t group_stride = 0) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(B12X_B200_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t dims[3] = {cols, rows, groups};
  // Elements between the same row of consecutive groups: group-major [L][rows][ld] by default.
  const cuuint64_t strides[2] = {ld * 2, (group_stride ? group_stride : rows * ld) * 2};
  const cuuint32_t box[3] = {box_cols, box_rows, 1};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  const CUresult r =
      fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(base), dims, strides, box,
         elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_last_error, sizeof(g_last_error), "cuTensorMapEncodeTiled(raw rows) failed (%d)", int(r));
    return B12X_B200_ERR_CUDA;
  }
  return B12X_B200_OK;
}

// Row-major 2-byte matrix [rows, cols] with row pitch `ld` elements -> boxes of 64 columns
// (128 bytes) x 128 rows, 128-byte swizzle; used for TMA stores of BF16/FP16 outputs.
inline int make_output_map_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols,
                       uint64_t ld) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(B12X_B200_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {ld * 2};
  const cuuint32_t box[2] = {64, 128};
  const cuuint32_t elem_strides[2] = {1, 1};
  const CUresult r =
      fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), dims, strides, box,
         elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
         CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_last_error, sizeof(g_last_error), "cuTensorMapEncodeTiled(C) failed (%d)", int(r));
    return B12X_B200_ERR_CUDA;
  }
  return B12X_B200_OK;
}

// The same for a stack of `groups` outputs [groups, rows, ld] (a store never spills into the
// next group: rows at or beyond `rows` are clipped).
inline int make_output_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                    uint64_t groups = 1) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(B12X_B200_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t dims[3] = {cols, rows, groups};
  const cuuint64_t strides[2] = {ld * 2, rows * ld * 2};
  const cuuint32_t box[3] = {64, 128, 1};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  const CUresult r =
      fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(base), dims, strides, box,
         elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
         CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_last_error, sizeof(g_last_error), "cuTensorMapEncodeTiled(C) failed (%d)", int(r));
    return B12X_B200_ERR_CUDA;
  }
  return B12X_B200_OK;
}

struct DeviceInfo {
  int sm_count = 0;
  int cc_major = 0;
};

inline int device_info(DeviceInfo* out) {
  static DeviceInfo cache[64];
  static bool have[64] = {};
  static std::mutex mu;
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) return fail_cuda(err, "cudaGetDevice");
  std::lock_guard<std::mutex> lock(mu);
  if (dev < 0 || dev >= 64) return fail(B12X_B200_ERR_INVALID_ARGUMENT, "device index out of range");
  if (!have[dev]) {
    err = cudaDeviceGetAttribute(&cache[dev].sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (err != cudaSuccess) return fail_cuda(err, "cudaDeviceGetAttribute");
    err = cudaDeviceGetAttribute(&cache[dev].cc_major, cudaDevAttrComputeCapabilityMajor, dev);
    if (err != cudaSuccess) return fail_cuda(err, "cudaDeviceGetAttribute");
    have[dev] = true;
  }
  *out = cache[dev];
  return B12X_B200_OK;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Experiment switches, read from the environment once per process (never on the launch path).
// They exist for measurements of kernel variants; none is part of the interface.
struct Switches {
  bool decode_overlap = true;   // programmatic stream serialization for decode GEMMs / quantizers
  bool pair_tail_split = true;  // split-K the last partial round of the CTA-pair kernel
  bool bmm_tensor_core = true;  // batched BF16 x MXFP8 product on warp-level MMAs when it fits
};

inline const Switches& switches() {
  static const Switches sw = [] {
    Switches v;
    if (const char* e = getenv("B12X_B200_DECODE_OVERLAP")) v.decode_overlap = atoi(e) != 0;
    if (const char* e = getenv("B12X_B200_PAIR_TAIL_SPLIT")) v.pair_tail_split = atoi(e) != 0;
    if (const char* e = getenv("B12X_B200_BMM_TENSOR_CORE")) v.bmm_tensor_core = atoi(e) != 0;
    return v;
  }();
  return sw;
}

// Rows up to which a quantized matrix is taken for an activation (its quantization releases the
// next kernel early) and a decode GEMM's weight for something a predecessor may just have
// written (its stream waits for the predecessor). One constant, so the two rules meet.
constexpr int kEarlyReleaseRows = 128;

// Workspace layout shared by the kernels that need scratch (one buffer per stream serves them
// all, launches on a stream being ordered): 60 KiB of per-tile counters of the decode kernel,
// 4 KiB of counters of the CTA-pair kernel's split tail, then FP32 partial tiles from 64 KiB on.
constexpr size_t kSmallMCounterBytes = 60 * 1024;
constexpr size_t kPairCounterOffset = kSmallMCounterBytes;
constexpr size_t kPairCounterBytes = 4 * 1024;
constexpr size_t kWorkspaceHeaderBytes = kPairCounterOffset + kPairCounterBytes;

}  // namespace b12x_b200
