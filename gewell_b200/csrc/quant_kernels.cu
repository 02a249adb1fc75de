// HBM-bound element-wise kernels of the quantised-projection path: weight
// dequantise / pack / fake-quant and activation quantisation (NVFP4 and FP8,
// with optional fused GeGLU).  All are pure streaming kernels: 16- or 32-byte
// vector accesses, one K16 block (or 16 FP8 values) per thread, eight values where GeGLU comes first.  A matrix is
// walked as slabs of whole 128-row groups (blockIdx.y) so that the index inside a slab fits the 31 bits of a
// multiply-high division; with 64-bit divisions the kernels were bound by index arithmetic, not by memory.
#include "common.cuh"
#include "kernels.h"

#include <cmath>

namespace gw {
namespace {

constexpr int kThreads = 256;

struct alignas(16) Bf16x8 { uint4 v; };

__device__ __forceinline__ void unpack8(const uint4& raw, float* out) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    out[2 * i] = __uint_as_float(w[i] << 16);
    out[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

// 128-row groups per slab, so that `per_row` items of each of its rows number less than 2^31.  `padding`: rows up to the next
// multiple of 128 have items too (scale tiles); without it a matrix of one slab has blocks for its own rows alone.
struct Slabs {
  uint32_t rows, count;
  Slabs(uint32_t total_rows, uint32_t per_row, bool padding) {
    const uint64_t fit = ((1ull << 31) - 1) / (uint64_t(per_row ? per_row : 1) * 128) * 128;
    const uint64_t all = padding ? (uint64_t(total_rows) + 127) / 128 * 128 : total_rows;
    rows = uint32_t(fit == 0 ? 128 : fit < all ? fit : all);
    count = uint32_t((all + rows - 1) / rows);
  }
};

// largest magnitude of packed BF16 values
template <int N>
__device__ __forceinline__ float absmax_words(const uint32_t (&w)[N]) {
  __nv_bfloat162 best = __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[0]));
#pragma unroll
  for (int i = 1; i < N; ++i) best = __hmax2(best, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));
  return fmaxf(0.0F, fmaxf(__low2float(best), __high2float(best)));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&pair);
}

// ---------------------------------------------------------------------------
// NVFP4 weight dequantise: one thread per K16 block (8 packed bytes in,
// 32 bytes of BF16 out).  Reference: src/nvfp4_linear.cu:39-56.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
nvfp4_dequantize_kernel(const uint8_t* __restrict__ data, const uint8_t* __restrict__ scales, float weight_scale, uint32_t width,
                        Divisor blocks_per_row, uint32_t slab_rows, uint32_t rows, uint4* __restrict__ output) {
  const uint32_t row0 = blockIdx.y * slab_rows;
  const uint32_t index = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t local = blocks_per_row.quotient(index), kb = index - local * blocks_per_row.value;
  if (local >= min(slab_rows, rows - row0)) return;
  const size_t row = row0 + size_t(local);
  const size_t block = row * blocks_per_row.value + kb;
  const float scale = __fmul_rn(e4m3_to_float(scales[scale_offset(row, kb, width)]), weight_scale);
  const uint2 packed = reinterpret_cast<const uint2*>(data)[block];
  const uint32_t words[2] = {packed.x, packed.y};
  uint32_t out[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 pair = e2m1x2_to_float2((words[i / 4] >> (8 * (i % 4))) & 0xFF);
    out[i] = pack_bf16x2(__fmul_rn(pair.x, scale), __fmul_rn(pair.y, scale));
  }
  output[2 * block] = make_uint4(out[0], out[1], out[2], out[3]);
  output[2 * block + 1] = make_uint4(out[4], out[5], out[6], out[7]);
}

// ---------------------------------------------------------------------------
// NVFP4 weight pack: tools/convert.py:111-137 / src/weight_qdq_detail.cuh:73-82.
// One thread per (row in the 128-padded grid, K16 block in the 4-padded grid)
// so that every byte of the scale storage is written (padding = 0).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
nvfp4_pack_weights_kernel(const uint4* __restrict__ weights, uint32_t rows, uint32_t width, float global_scale,
                          uint2* __restrict__ data, uint8_t* __restrict__ scales, Divisor padded_blocks_per_row, uint32_t slab_rows) {
  const uint32_t index = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t local = padded_blocks_per_row.quotient(index), kb = index - local * padded_blocks_per_row.value;
  if (local >= slab_rows) return;
  const size_t row = size_t(blockIdx.y) * slab_rows + local;
  if (row >= (size_t(rows) + 127) / 128 * 128) return;
  const uint32_t blocks_per_row = width / 16;
  uint8_t scale_code = 0;
  if (row < rows && kb < blocks_per_row) {
    const size_t block = row * blocks_per_row + kb;
    float values[16];
    unpack8(weights[2 * block], values);
    unpack8(weights[2 * block + 1], values + 8);
    float amax = 0.0F;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(values[i]));
    float unrounded = 1.0F;
    if (amax != 0.0F)
      unrounded = fminf(448.0F, fmaxf(0x1p-9F, __fdiv_rn(amax, __fmul_rn(6.0F, global_scale))));
    scale_code = float_to_e4m3(unrounded);
    const float decoded = __fmul_rn(e4m3_to_float(scale_code), global_scale);
    uint32_t words[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t byte = float2_to_e2m1x2(__fdiv_rn(values[2 * i], decoded),
                                             __fdiv_rn(values[2 * i + 1], decoded));
      words[i / 4] |= byte << (8 * (i % 4));
    }
    data[block] = make_uint2(words[0], words[1]);
  }
  scales[scale_offset(row, kb, width)] = scale_code;
}

// ---------------------------------------------------------------------------
// NVFP4 activation quantise (+GeGLU): src/nvfp4_linear.cu:61-116.  The three
// approximate reciprocals and the FP32 multiply order are the reference's.
// A K16 block is one thread's, or two threads' with GeGLU in front (sixteen unrolled tanh are bound by fetching
// the code at decode sizes); the threads of a 64-value group put their scale codes together and one of them
// stores four bytes.  Entries outside [rows, K/16] are the zero padding of the scale tiles.
// ---------------------------------------------------------------------------
template <bool Gelu>
__global__ void __launch_bounds__(kThreads)
nvfp4_quantize_kernel(const uint4* __restrict__ input, uint32_t rows, uint32_t width, float inverse_global_scale,
                      uint32_t* __restrict__ packed, uint8_t* __restrict__ scales, Divisor padded_items_per_row, uint32_t slab_rows) {
  constexpr int kWords = Gelu ? 4 : 8;          // packed BF16 pairs per thread
  constexpr int kShare = 8 / kWords;            // threads per K16 block
  griddep_enter_first();   // the GEMM that follows may set itself up while this kernel waits
  // items of a row: a multiple of 4 * kShare, so whole K64 groups are inside or outside and sit in one warp
  const uint32_t index = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t local = padded_items_per_row.quotient(index), item = index - local * padded_items_per_row.value;
  const size_t row = size_t(blockIdx.y) * slab_rows + local;
  const bool tile = local < slab_rows && row < (size_t(rows) + 127) / 128 * 128;
  const uint32_t items_per_row = width / (2 * kWords);
  const bool live = tile && row < rows && item < items_per_row;
  uint32_t scale_code = 0;
  uint32_t words[kWords] = {};
  if (live) {
    if constexpr (Gelu) {
      // input is [rows, 2K]: gate slice then up slice
      const uint4 gate = input[row * (2 * size_t(items_per_row)) + item], up = input[row * (2 * size_t(items_per_row)) + items_per_row + item];
      float g[8], u[8];
      unpack8(gate, g);
      unpack8(up, u);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        words[i] = (__float_as_uint(gelu_tanh_multiply_bf16(g[2 * i], u[2 * i])) >> 16) |
                   (__float_as_uint(gelu_tanh_multiply_bf16(g[2 * i + 1], u[2 * i + 1])) & 0xFFFF0000u);
    } else {
      const uint4* source = input + 2 * (row * items_per_row + item);
      const uint4 lo = source[0], hi = source[1];
      words[0] = lo.x; words[1] = lo.y; words[2] = lo.z; words[3] = lo.w;
      words[4] = hi.x; words[5] = hi.y; words[6] = hi.z; words[7] = hi.w;
    }
  }
  float amax = absmax_words(words);
  if constexpr (kShare == 2) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  if (live) {
    scale_code = float_to_e4m3(inverse_global_scale * (amax * rcp_approx_ftz(6.0F)));
    const float block_scale = e4m3_to_float(uint8_t(scale_code));
    const float factor = block_scale == 0.0F
                             ? 0.0F
                             : rcp_approx_ftz(block_scale * rcp_approx_ftz(inverse_global_scale));
    uint32_t out[kWords / 4] = {};
#pragma unroll
    for (int i = 0; i < kWords; ++i)
      out[i / 4] |= uint32_t(float2_to_e2m1x2(__uint_as_float(words[i] << 16) * factor, __uint_as_float(words[i] & 0xFFFF0000u) * factor)) << (8 * (i % 4));
    const size_t at = row * items_per_row + item;
    if constexpr (Gelu) packed[at] = out[0];
    else reinterpret_cast<uint2*>(packed)[at] = make_uint2(out[0], out[1]);
  }
  // byte kb % 4 of the word that the K64 group's first thread stores
  uint32_t word = scale_code;
  word |= __shfl_down_sync(0xffffffffu, word, kShare) << 8;
  word |= __shfl_down_sync(0xffffffffu, word, 2 * kShare) << 16;
  if (!tile) return;
  if (reinterpret_cast<uintptr_t>(scales) % 4 == 0) {
    if (item % (4 * kShare) == 0) *reinterpret_cast<uint32_t*>(scales + scale_offset(row, item / kShare, width)) = word;
  } else if (item % kShare == 0) {
    scales[scale_offset(row, item / kShare, width)] = uint8_t(scale_code);
  }
}

// ---------------------------------------------------------------------------
// FP8 activation quantise (+GeGLU): src/fp8_linear.cu:33-52.  16 values per thread, eight with GeGLU in front.
// width % 16 == 0 keeps rows 16-byte aligned when the input pointer is; a 2-byte-aligned input takes scalar loads.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t fp8_words(float a, float b, float c, float d, float inverse_scale) {
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(__fmul_rn(a, inverse_scale), __fmul_rn(b, inverse_scale)), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(__fmul_rn(c, inverse_scale), __fmul_rn(d, inverse_scale)), __NV_SATFINITE, __NV_E4M3);
  return lo | hi << 16;
}
template <bool Vector>
__device__ __forceinline__ void load8(const bf16* src, float* dst) {
  if constexpr (Vector) {
    unpack8(*reinterpret_cast<const uint4*>(src), dst);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[i] = __bfloat162float(src[i]);
  }
}
template <bool Gelu, bool Vector>
__global__ void __launch_bounds__(kThreads)
fp8_quantize_kernel(const bf16* __restrict__ input, uint32_t rows, uint32_t width, Divisor items_per_row, uint32_t slab_rows,
                    float inverse_scale, uint8_t* __restrict__ packed) {
  constexpr uint32_t kValues = Gelu ? 8 : 16;
  griddep_enter_first();   // the GEMM that follows may set itself up while this kernel waits
  const uint32_t row0 = blockIdx.y * slab_rows;
  const uint32_t index = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t local = items_per_row.quotient(index), col = (index - local * items_per_row.value) * kValues;
  if (local >= min(slab_rows, rows - row0)) return;
  const size_t row = row0 + size_t(local);
  float values[kValues];
  if constexpr (Gelu) {
    float g[8], u[8];
    load8<Vector>(input + row * 2 * width + col, g);
    load8<Vector>(input + row * 2 * width + width + col, u);
#pragma unroll
    for (int i = 0; i < 8; ++i) values[i] = gelu_tanh_multiply_bf16(g[i], u[i]);
  } else {
    load8<Vector>(input + row * width + col, values);
    load8<Vector>(input + row * width + col + 8, values + 8);
  }
  uint32_t words[kValues / 4];
#pragma unroll
  for (uint32_t i = 0; i < kValues / 4; ++i)
    words[i] = fp8_words(values[4 * i], values[4 * i + 1], values[4 * i + 2], values[4 * i + 3], inverse_scale);
  uint8_t* out = packed + row * width + col;
  if constexpr (Gelu) {
    *reinterpret_cast<uint2*>(out) = make_uint2(words[0], words[1]);
  } else if (reinterpret_cast<uintptr_t>(packed) % 16 == 0) {
    *reinterpret_cast<uint4*>(out) = make_uint4(words[0], words[1], words[2], words[3]);
  } else {
    reinterpret_cast<uint2*>(out)[0] = make_uint2(words[0], words[1]);
    reinterpret_cast<uint2*>(out)[1] = make_uint2(words[2], words[3]);
  }
}

// FP8 weight pack: tools/convert.py:49-62 (code = e4m3(x / scale)).
__global__ void __launch_bounds__(kThreads)
fp8_pack_weights_kernel(const uint4* __restrict__ weights, size_t groups, uint32_t width, float scale,
                        const float* __restrict__ row_scales, uint2* __restrict__ data) {
  for (size_t group = size_t(blockIdx.x) * kThreads + threadIdx.x; group < groups;
       group += size_t(gridDim.x) * kThreads) {
    const float s = row_scales ? row_scales[group / (width / 8)] : scale;
    float values[8];
    unpack8(weights[group], values);
    uint32_t words[2] = {0, 0};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t pair = __nv_cvt_float2_to_fp8x2(
          make_float2(__fdiv_rn(values[2 * i], s), __fdiv_rn(values[2 * i + 1], s)), __NV_SATFINITE,
          __NV_E4M3);
      words[i / 2] |= pair << (16 * (i % 2));
    }
    data[group] = make_uint2(words[0], words[1]);
  }
}

// ---------------------------------------------------------------------------
// Weight QDQ: src/weight_qdq.cu:105-189.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
absmax_kernel(const bf16* __restrict__ values, uint64_t elements, uint32_t* __restrict__ state) {
  float local = 0.0F;
  bool bad = false;
  const auto look = [&](float v) {
    if (!isfinite(v)) bad = true; else local = fmaxf(local, fabsf(v));
  };
  // 16-byte loads over the whole vectors of an aligned tensor, single values for the rest
  const uint64_t vectors = reinterpret_cast<uintptr_t>(values) % 16 == 0 ? elements / 8 : 0;
  const uint64_t first = uint64_t(blockIdx.x) * kThreads + threadIdx.x, step = uint64_t(gridDim.x) * kThreads;
#pragma unroll 4
  for (uint64_t i = first; i < vectors; i += step) {
    float v[8];
    unpack8(reinterpret_cast<const uint4*>(values)[i], v);
#pragma unroll
    for (int e = 0; e < 8; ++e) look(v[e]);
  }
  for (uint64_t i = vectors * 8 + first; i < elements; i += step) look(__bfloat162float(values[i]));
  for (int offset = 16; offset; offset /= 2)
    local = fmaxf(local, __shfl_xor_sync(0xffffffffu, local, offset));
  bad = __any_sync(0xffffffffu, bad);
  __shared__ float warp_max[kThreads / 32];
  __shared__ int warp_bad[kThreads / 32];
  if (threadIdx.x % 32 == 0) { warp_max[threadIdx.x / 32] = local; warp_bad[threadIdx.x / 32] = bad; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 0; w < kThreads / 32; ++w) { local = fmaxf(local, warp_max[w]); bad |= warp_bad[w] != 0; }
    atomicMax(state, __float_as_uint(local));   // non-negative floats order like their bits
    if (bad) atomicExch(state + 1, 1u);
  }
}

__global__ void __launch_bounds__(kThreads)
fp8_qdq_kernel(bf16* __restrict__ values, uint64_t elements, float scale) {
  const auto qdq = [&](float v) { return __fmul_rn(e4m3_to_float(float_to_e4m3(__fdiv_rn(v, scale))), scale); };
  const uint64_t vectors = reinterpret_cast<uintptr_t>(values) % 16 == 0 ? elements / 8 : 0;
  const uint64_t first = uint64_t(blockIdx.x) * kThreads + threadIdx.x, step = uint64_t(gridDim.x) * kThreads;
  for (uint64_t i = first; i < vectors; i += step) {
    float v[8];
    unpack8(reinterpret_cast<const uint4*>(values)[i], v);
    uint32_t words[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) words[e] = pack_bf16x2(qdq(v[2 * e]), qdq(v[2 * e + 1]));
    reinterpret_cast<uint4*>(values)[i] = make_uint4(words[0], words[1], words[2], words[3]);
  }
  for (uint64_t i = vectors * 8 + first; i < elements; i += step) values[i] = __float2bfloat16_rn(qdq(__bfloat162float(values[i])));
}

// value / divisor, correctly rounded.  A zero numerator takes the division's slow path, and the whole warp waits for it: weights
// that went through FP4 before are a quarter zeros.  So zeros divide something else, and their quotient is themselves.
// (82 M such values 136 -> 60 us.  The packers, whose input is seldom zero, are slower by the selection: 55 -> 63 us.)
__device__ __forceinline__ float divide(float value, float divisor) {
  const float q = __fdiv_rn(value == 0.0F ? divisor : value, divisor);
  return value == 0.0F && divisor > 0.0F ? value : q;
}

// One thread per K16 block of the flat tensor (32-byte load and store).
__global__ void __launch_bounds__(kThreads)
nvfp4_qdq_kernel(uint4* __restrict__ values, uint64_t blocks, float global_scale) {
  for (uint64_t block = uint64_t(blockIdx.x) * kThreads + threadIdx.x; block < blocks;
       block += uint64_t(gridDim.x) * kThreads) {
    float v[16];
    unpack8(values[2 * block], v);
    unpack8(values[2 * block + 1], v + 8);
    float amax = 0.0F;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
    float block_scale = 1.0F;
    if (amax != 0.0F) {
      const float clamped =
          fminf(448.0F, fmaxf(0x1p-9F, __fdiv_rn(amax, __fmul_rn(6.0F, global_scale))));
      block_scale = e4m3_to_float(float_to_e4m3(clamped));
    }
    const float combined = __fmul_rn(block_scale, global_scale);
    uint32_t out[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 q = e2m1x2_to_float2(
          float2_to_e2m1x2(divide(v[2 * i], combined), divide(v[2 * i + 1], combined)));
      out[i] = pack_bf16x2(__fmul_rn(q.x, combined), __fmul_rn(q.y, combined));
    }
    values[2 * block] = make_uint4(out[0], out[1], out[2], out[3]);
    values[2 * block + 1] = make_uint4(out[4], out[5], out[6], out[7]);
  }
}

__global__ void rcp_approx_kernel(const float* __restrict__ in, float* __restrict__ out, size_t n) {
  const size_t i = size_t(blockIdx.x) * kThreads + threadIdx.x;
  if (i < n) out[i] = rcp_approx_ftz(in[i]);
}

__device__ __forceinline__ uint4 geglu8(const uint4& g, const uint4& u) {
  const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
  uint32_t words[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float a = gelu_tanh_multiply_bf16(__uint_as_float(gw[k] << 16), __uint_as_float(uw[k] << 16));
    const float b = gelu_tanh_multiply_bf16(__uint_as_float(gw[k] & 0xFFFF0000u), __uint_as_float(uw[k] & 0xFFFF0000u));
    words[k] = (__float_as_uint(a) >> 16) | (__float_as_uint(b) & 0xFFFF0000u);
  }
  return make_uint4(words[0], words[1], words[2], words[3]);
}

// VECTOR: 16-byte aligned buffers, eight values a thread (the last thread takes what is left)
template <bool VECTOR>
__global__ void geglu_kernel(const bf16* gate, const bf16* up, bf16* out, size_t n) {
  griddep_enter();
  const size_t i = (size_t(blockIdx.x) * kThreads + threadIdx.x) * (VECTOR ? 8 : 1);
  if (VECTOR && i + 8 <= n) {
    *reinterpret_cast<uint4*>(out + i) = geglu8(*reinterpret_cast<const uint4*>(gate + i), *reinterpret_cast<const uint4*>(up + i));
  } else {
#pragma unroll 1
    for (size_t j = i; j < n && j < i + (VECTOR ? 8 : 1); ++j)
      out[j] = __float2bfloat16_rn(gelu_tanh_multiply_bf16(__bfloat162float(gate[j]), __bfloat162float(up[j])));
  }
}

// [rows, gate | up] -> [rows, width]: eight channels per thread, 16-byte loads and stores
__global__ void geglu_interleaved_kernel(const uint4* __restrict__ gate_up, uint4* __restrict__ out, Divisor row_vectors,
                                         uint32_t slab_rows, uint32_t rows) {
  griddep_enter();
  const uint32_t row0 = blockIdx.y * slab_rows, index = blockIdx.x * kThreads + threadIdx.x;
  const uint32_t local = row_vectors.quotient(index), v = index - local * row_vectors.value;
  if (local >= min(slab_rows, rows - row0)) return;
  const size_t row = row0 + size_t(local), vectors = row_vectors.value;
  out[row * vectors + v] = geglu8(gate_up[row * 2 * vectors + v], gate_up[row * 2 * vectors + vectors + v]);
}

unsigned grid_for(size_t items, size_t cap = 1u << 20) {
  size_t blocks = (items + kThreads - 1) / kThreads;
  if (blocks < 1) blocks = 1;
  if (blocks > cap) blocks = cap;
  return static_cast<unsigned>(blocks);
}

}  // namespace

namespace {
dim3 slab_grid(const Slabs& slabs, uint32_t per_row) {
  return dim3(unsigned((uint64_t(slabs.rows) * per_row + kThreads - 1) / kThreads), slabs.count);
}
}  // namespace

cudaError_t launch_nvfp4_dequantize(const uint8_t* data, const uint8_t* scales, float weight_scale,
                                    uint32_t width, uint32_t rows, void* output, cudaStream_t stream) {
  const uint32_t per_row = width / 16;
  const Slabs slabs(rows, per_row, false);
  nvfp4_dequantize_kernel<<<slab_grid(slabs, per_row), kThreads, 0, stream>>>(data, scales, weight_scale, width, Divisor::of(per_row),
                                                                             slabs.rows, rows, static_cast<uint4*>(output));
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_nvfp4_pack_weights(const void* weights, uint32_t rows, uint32_t width,
                                      float weight_scale, uint8_t* data, uint8_t* scales,
                                      cudaStream_t stream) {
  const uint32_t per_row = (width + 63) / 64 * 4;
  const Slabs slabs(rows, per_row, true);
  nvfp4_pack_weights_kernel<<<slab_grid(slabs, per_row), kThreads, 0, stream>>>(
      static_cast<const uint4*>(weights), rows, width, weight_scale, reinterpret_cast<uint2*>(data), scales, Divisor::of(per_row), slabs.rows);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_nvfp4_quantize(const void* input, uint32_t rows, uint32_t width,
                                  float inverse_global_scale, bool gelu, uint8_t* packed,
                                  uint8_t* scales, cudaStream_t stream) {
  const uint32_t per_row = (width + 63) / 64 * (gelu ? 8 : 4);
  const Slabs slabs(rows, per_row, true);
  return launch_pdl(gelu ? nvfp4_quantize_kernel<true> : nvfp4_quantize_kernel<false>, slab_grid(slabs, per_row), kThreads, stream,
                    static_cast<const uint4*>(input), rows, width, inverse_global_scale, reinterpret_cast<uint32_t*>(packed), scales,
                    Divisor::of(per_row), slabs.rows);
}

cudaError_t launch_fp8_quantize(const void* input, uint32_t rows, uint32_t width, float inverse_scale,
                                bool gelu, uint8_t* packed, cudaStream_t stream) {
  const bool vector = reinterpret_cast<uintptr_t>(input) % 16 == 0;
  const uint32_t per_row = width / (gelu ? 8 : 16);
  const Slabs slabs(rows, per_row, false);
  const auto kernel = gelu ? (vector ? fp8_quantize_kernel<true, true> : fp8_quantize_kernel<true, false>)
                           : (vector ? fp8_quantize_kernel<false, true> : fp8_quantize_kernel<false, false>);
  return launch_pdl(kernel, slab_grid(slabs, per_row), kThreads, stream, static_cast<const bf16*>(input), rows, width, Divisor::of(per_row),
                    slabs.rows, inverse_scale, packed);
}

cudaError_t launch_fp8_pack_weights(const void* weights, uint32_t rows, uint32_t width, float scale,
                                    const float* row_scales, uint8_t* data, cudaStream_t stream) {
  const size_t groups = size_t(rows) * (width / 8);
  fp8_pack_weights_kernel<<<grid_for(groups, 148 * 32), kThreads, 0, stream>>>(
      static_cast<const uint4*>(weights), groups, width, scale, row_scales, reinterpret_cast<uint2*>(data));
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_rcp_approx(const float* in, float* out, size_t n, cudaStream_t stream) {
  rcp_approx_kernel<<<grid_for(n, ~0u), kThreads, 0, stream>>>(in, out, n);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_geglu(const void* gate, const void* up, void* out, size_t n, cudaStream_t stream) {
  const auto off = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 != 0; };
  const bool vector = !off(gate) && !off(up) && !off(out);
  return launch_pdl(vector ? geglu_kernel<true> : geglu_kernel<false>, grid_for(vector ? (n + 7) / 8 : n, ~0u), kThreads, stream,
                    static_cast<const bf16*>(gate), static_cast<const bf16*>(up), static_cast<bf16*>(out), n);
}

cudaError_t launch_geglu_interleaved(const void* gate_up, void* out, uint32_t rows, uint32_t width, cudaStream_t stream) {
  const Slabs slabs(rows, width / 8, false);
  return launch_pdl(geglu_interleaved_kernel, slab_grid(slabs, width / 8), kThreads, stream, static_cast<const uint4*>(gate_up),
                    static_cast<uint4*>(out), Divisor::of(width / 8), slabs.rows, rows);
}

cudaError_t launch_absmax(const void* values, uint64_t elements, uint32_t* state, cudaStream_t stream) {
  cudaError_t status = cudaMemsetAsync(state, 0, 2 * sizeof(uint32_t), stream);
  if (status != cudaSuccess) return status;
  absmax_kernel<<<grid_for((elements + 7) / 8, 148 * 8), kThreads, 0, stream>>>(
      static_cast<const bf16*>(values), elements, state);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_fp8_qdq(void* values, uint64_t elements, float scale, cudaStream_t stream) {
  fp8_qdq_kernel<<<grid_for((elements + 7) / 8, 148 * 32), kThreads, 0, stream>>>(static_cast<bf16*>(values), elements, scale);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_nvfp4_qdq(void* values, uint64_t elements, float global_scale, cudaStream_t stream) {
  nvfp4_qdq_kernel<<<grid_for(elements / 16, 148 * 64), kThreads, 0, stream>>>(
      static_cast<uint4*>(values), elements / 16, global_scale);
  note_launch();
  return cudaGetLastError();
}

}  // namespace gw
