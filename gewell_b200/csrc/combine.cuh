// The weighted sum of a token's expert rows: eight BF16 values per thread.
#pragma once

#include "common.cuh"

namespace gw {

// Row j contributes bf16(value * weight), added in BF16 by ascending j.  All gathered loads are in flight before the
// fold starts; each of the rows is read once in the layer.
template <int ROWS>
__device__ __forceinline__ uint4 combine_rows(const uint4* __restrict__ down, const int32_t* rows, const float* weights, uint32_t vectors,
                                              uint32_t v) {
  uint4 raw[ROWS];
#pragma unroll
  for (int j = 0; j < ROWS; ++j) raw[j] = __ldcs(down + size_t(rows[j]) * vectors + v);
  __nv_bfloat162 sum[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) sum[i] = __floats2bfloat162_rn(0.0F, 0.0F);
#pragma unroll
  for (int j = 0; j < ROWS; ++j) {
    const float w = weights[j];
    const uint32_t words[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 product = __floats2bfloat162_rn(__fmul_rn(__uint_as_float(words[i] << 16), w),
                                                           __fmul_rn(__uint_as_float(words[i] & 0xFFFF0000u), w));
      sum[i] = __hadd2(sum[i], product);
    }
  }
  return make_uint4(*reinterpret_cast<const uint32_t*>(&sum[0]), *reinterpret_cast<const uint32_t*>(&sum[1]),
                    *reinterpret_cast<const uint32_t*>(&sum[2]), *reinterpret_cast<const uint32_t*>(&sum[3]));
}

}  // namespace gw
