// Output of the weight-streaming kernels: a warp turns eight rows x 32 columns around in shared
// memory and stores 16 bytes per lane.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "gemm_blockscaled.cuh"

namespace b12x_b200 {

// Eight consecutive output rows x this warp's 32 columns, one value per row in each lane:
// turned around in the warp's 512 bytes of staging memory and stored as 16 bytes per lane (lane
// l: row l / 4, columns (l % 4) * 8 .. + 7). `vals` are final values (scaled); rows from
// `row0 + 8` on or beyond `m`, and columns beyond `n`, are not written. `P` names the output: c,
// m, n, ldc, out_dtype (2-byte types).
template <typename P>
__device__ __forceinline__ void store_rows8_packed(const P& p, uint16_t* buf, int lane,
                                                   size_t c_group0, int row0, int col0,
                                                   const float (&vals)[8]) {
  __syncwarp();  // the previous eight rows have been read
#pragma unroll
  for (int r = 0; r < 8; ++r)
    buf[r * 32 + lane] = (p.out_dtype == kOutBf16) ? __bfloat16_as_ushort(__float2bfloat16_rn(vals[r]))
                                                   : __half_as_ushort(__float2half_rn(vals[r]));
  __syncwarp();
  const int r8 = lane >> 2;
  const int j4 = lane & 3;
  const int mrow = row0 + r8;
  const int col = col0 + j4 * 8;
  if (mrow < p.m && col < p.n) {
    uint16_t* dst = static_cast<uint16_t*>(p.c) + c_group0 + static_cast<size_t>(mrow) * p.ldc + col;
    if (col + 8 <= p.n) {
      *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(buf + r8 * 32 + j4 * 8);
    } else {
      for (int e = 0; col + e < p.n; ++e) dst[e] = buf[r8 * 32 + j4 * 8 + e];
    }
  }
}

}  // namespace b12x_b200
