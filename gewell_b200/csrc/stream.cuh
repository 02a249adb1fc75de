// Device side of the weight-streaming projections (decode_stream.cu): how one warp multiplies a piece of
// 32 weight rows that lies in shared memory with up to 16 token rows.
//
// A piece is 32 rows x 128 bytes of K (256 E2M1, 128 E4M3 or 64 BF16 values of every row), as one tensor
// copy with the 128-byte swizzle leaves it: four groups ("slots" 0..3) of eight rows.  Lane 4 * g + t takes
// the 32 bytes t of row g of every slot.  Slots 0 and 1 are the rows g and g + 8 of one m16 tensor tile,
// slots 2 and 3 of a second.
//
// The tensor instruction is mma.sync m16n8k16 with FP32 accumulation.  Which sixteen K values make up
// a step is free as long as both operands agree: a step takes four consecutive values of every lane's
// own 32 bytes, so no value changes lanes.  With one to sixteen token columns the tensor instruction is not
// what bounds a launch; tcgen05 would want quantised tokens from a launch before and a tensor-memory prologue,
// and cannot take NVFP4 weights with BF16 activations at all.
//
// Both operands are exact: E2M1 x E4M3 block scale has six significant bits and fits FP16 (range
// 2^-10 .. 2688) as well as BF16, E4M3 fits FP16.  FP4 and FP8 activations are quantised by the same
// recipe as everywhere else and kept as codes in shared memory, BF16 activations as they are.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"
#include "decode_stream.h"
#include "ptx.cuh"

namespace gw::stream {

constexpr uint32_t kPieceBytes = 32 * 128;
constexpr uint32_t kPieceScaleBytes = 512;      // NVFP4: four block scales of every row

// lane_values: K values in a lane's 32 bytes
__host__ __device__ constexpr int lane_values(StreamKind kind) {
  return kind == StreamKind::w16a16 ? 16 : kind == StreamKind::w8a8 ? 32 : 64;
}
__host__ __device__ constexpr int chunk_values(StreamKind kind) { return 4 * lane_values(kind); }
__host__ __device__ constexpr bool nvfp4_weights(StreamKind kind) {
  return kind == StreamKind::w4a4 || kind == StreamKind::w4a16;
}
// 16-byte vectors of token values (eight 16-bit values) that a lane needs per piece and token group
__host__ __device__ constexpr int token_vectors(StreamKind kind) { return lane_values(kind) / 8; }

__device__ __forceinline__ void mma_f16(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// four bytes = eight E2M1 values -> four FP16 pairs in K order
__device__ __forceinline__ void e2m1x8_to_f16(uint32_t word, uint32_t* r) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\tcvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\tcvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(word));
}
// four bytes = four E4M3 values -> two FP16 pairs
__device__ __forceinline__ void e4m3x4_to_f16(uint32_t word, uint32_t* r) {
  asm("{\n\t.reg .b16 h0, h1;\n\tmov.b32 {h0, h1}, %2;\n\t"
      "cvt.rn.f16x2.e4m3x2 %0, h0;\n\tcvt.rn.f16x2.e4m3x2 %1, h1;\n\t}" : "=r"(r[0]), "=r"(r[1]) : "r"(word));
}
__device__ __forceinline__ uint32_t mul_f16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

// W4A16.  An E2M1 code's three magnitude bits, put at bits 8..6 of a BF16 pattern, are the value times
// 2^-126 (the code for 0.5 lands on a subnormal, as it is one in E2M1 too); multiplying by the block scale
// times 2^118 gives value x scale x 2^-8 exactly, and the epilogue's multiplier carries the 2^8.  A multiplication puts the
// sign and the magnitude of a pair of nibbles in their places at once, which leaves nine instructions of eight codes to the
// ALU, the pipe that bounds the kernel, instead of twelve (MLP of one row 63.0 -> 59.8 us).  Nibbles j
// and j + 4 of a word share their shifts, so a pair holds values j and j + 4 (the tokens are stored in the
// same order).
constexpr float kW4a16Exponent = 0x1p118F;
constexpr float kW4a16Alpha = 256.0F;
__device__ __forceinline__ void e2m1x8_to_bf16(uint32_t word, uint32_t* r) {
  const uint32_t high = word >> 8;
  r[0] = ((word & 0x000F000Fu) * 0x1040u) & 0x81C081C0u;       // x << 12 for the sign, x << 6 for the magnitude
  r[1] = ((word & 0x00F000F0u) * 0x0104u) & 0x81C081C0u;
  r[2] = ((high & 0x000F000Fu) * 0x1040u) & 0x81C081C0u;
  r[3] = ((high & 0x00F000F0u) * 0x0104u) & 0x81C081C0u;
}

// two E4M3 block scales (the low half of the word) -> one pair (s, s) per scale, in the format of the kind's multiplication
template <StreamKind KIND>
__device__ __forceinline__ void expand_scales(uint32_t word, uint32_t* r) {
  uint32_t h;
  asm("{\n\t.reg .b16 h0, h1;\n\tmov.b32 {h0, h1}, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, h0;\n\t}" : "=r"(h) : "r"(word));
  if constexpr (KIND == StreamKind::w4a4) {
    r[0] = __byte_perm(h, 0, 0x1010);
    r[1] = __byte_perm(h, 0, 0x3232);
  } else {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    r[0] = __byte_perm(__float_as_uint(f.x * kW4a16Exponent), 0, 0x3232);        // exact: four significant bits
    r[1] = __byte_perm(__float_as_uint(f.y * kW4a16Exponent), 0, 0x3232);
  }
}

// Token values of a chunk and eight tokens, `chunk_bytes`: FP4 codes or E4M3 codes [16-byte half][lane] and, FP4, one
// word of four block scales per lane; BF16 values [16-byte vector][lane].  Lane 4 * (token % 8) + t holds what
// the same lane of a weight row holds.
template <StreamKind KIND>
__host__ __device__ constexpr uint32_t token_chunk_bytes() {
  return KIND == StreamKind::w4a4 ? 1024 + 128 : KIND == StreamKind::w8a8 ? 1024 : lane_values(KIND) * 64;
}
// acc[tile of 16 rows][token group][4] += piece x tokens.  `piece`: shared-memory address of its weights plus
// the lane's row (g * 128); `scale_words`: the lane's block scales of the four slots, four each; `tokens`: shared-memory
// address of this chunk's token values (eight tokens after eight tokens).
template <StreamKind KIND, int NT>
__device__ __forceinline__ void multiply(uint32_t piece, uint32_t lane, const uint32_t* scale_words, uint32_t tokens,
                                         float (*acc)[NT][4]) {
  constexpr int kVectorsPerHalf = token_vectors(KIND) / 2;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t scale[4][2], token_scale[NT][2];
    if constexpr (nvfp4_weights(KIND)) {
#pragma unroll
      for (int q = 0; q < 4; ++q) expand_scales<KIND>(scale_words[q] >> (16 * half), scale[q]);
    }
    if constexpr (KIND == StreamKind::w4a4) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        expand_scales<KIND>(ptx::lds32(tokens + nt * token_chunk_bytes<KIND>() + 1024 + lane * 4) >> (16 * half), token_scale[nt]);
    }
    const uint32_t unit = (((lane % 4) * 2 + half) ^ (lane / 4)) * 16;
    uint4 w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = ptx::lds128(piece + q * 1024 + unit);
    uint4 codes[NT];
    if constexpr (KIND == StreamKind::w4a4 || KIND == StreamKind::w8a8) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) codes[nt] = ptx::lds128(tokens + nt * token_chunk_bytes<KIND>() + half * 512 + lane * 16);
    }
#pragma unroll
    for (int v = 0; v < kVectorsPerHalf; ++v) {
      const int vector = half * kVectorsPerHalf + v;
      uint32_t b[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const uint32_t c[4] = {codes[nt].x, codes[nt].y, codes[nt].z, codes[nt].w};
        if constexpr (KIND == StreamKind::w4a4) {
          e2m1x8_to_f16(c[v], b[nt]);
#pragma unroll
          for (int j = 0; j < 4; ++j) b[nt][j] = mul_f16x2(b[nt][j], token_scale[nt][v / 2]);
        } else if constexpr (KIND == StreamKind::w8a8) {
          e4m3x4_to_f16(c[2 * v], b[nt]);
          e4m3x4_to_f16(c[2 * v + 1], b[nt] + 2);
        } else {
          const uint4 x = ptx::lds128(tokens + nt * token_chunk_bytes<KIND>() + vector * 512 + lane * 16);
          b[nt][0] = x.x; b[nt][1] = x.y; b[nt][2] = x.z; b[nt][3] = x.w;
        }
      }
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        uint32_t lo[4], hi[4];        // rows g and g + 8: four pairs of K values = two steps
        const uint32_t lw[4] = {w[2 * mt].x, w[2 * mt].y, w[2 * mt].z, w[2 * mt].w};
        const uint32_t hw[4] = {w[2 * mt + 1].x, w[2 * mt + 1].y, w[2 * mt + 1].z, w[2 * mt + 1].w};
        if constexpr (nvfp4_weights(KIND)) {
          if constexpr (KIND == StreamKind::w4a4) {
            e2m1x8_to_f16(lw[v], lo);
            e2m1x8_to_f16(hw[v], hi);
          } else {
            e2m1x8_to_bf16(lw[v], lo);
            e2m1x8_to_bf16(hw[v], hi);
          }
          const uint32_t ls = scale[2 * mt][v / 2], hs = scale[2 * mt + 1][v / 2];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            lo[j] = KIND == StreamKind::w4a4 ? mul_f16x2(lo[j], ls) : mul_bf16x2(lo[j], ls);
            hi[j] = KIND == StreamKind::w4a4 ? mul_f16x2(hi[j], hs) : mul_bf16x2(hi[j], hs);
          }
        } else if constexpr (KIND == StreamKind::w8a8) {
          e4m3x4_to_f16(lw[2 * v], lo);
          e4m3x4_to_f16(lw[2 * v + 1], lo + 2);
          e4m3x4_to_f16(hw[2 * v], hi);
          e4m3x4_to_f16(hw[2 * v + 1], hi + 2);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            lo[j] = lw[j];
            hi[j] = hw[j];
          }
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          if constexpr (KIND == StreamKind::w4a4 || KIND == StreamKind::w8a8) {
            mma_f16(acc[mt][nt], lo[0], hi[0], lo[1], hi[1], b[nt][0], b[nt][1]);
            mma_f16(acc[mt][nt], lo[2], hi[2], lo[3], hi[3], b[nt][2], b[nt][3]);
          } else {
            mma_bf16(acc[mt][nt], lo[0], hi[0], lo[1], hi[1], b[nt][0], b[nt][1]);
            mma_bf16(acc[mt][nt], lo[2], hi[2], lo[3], hi[3], b[nt][2], b[nt][3]);
          }
        }
      }
    }
  }
}

// FP4 quantisation of sixteen activations, eight BF16 pairs (src/nvfp4_linear.cu:61-116): eight code bytes and the E4M3
// scale.  The maximum is taken on pairs; it is exact either way.
__device__ __forceinline__ uint8_t quantise_fp4(const uint32_t* pairs, float inverse_scale, uint32_t* codes) {
  const auto pair = [&](int i) { return __habs2(*reinterpret_cast<const __nv_bfloat162*>(pairs + i)); };
  const __nv_bfloat162 m = __hmax2(__hmax2(__hmax2(pair(0), pair(1)), __hmax2(pair(2), pair(3))),
                                   __hmax2(__hmax2(pair(4), pair(5)), __hmax2(pair(6), pair(7))));
  const float amax = fmaxf(__low2float(m), __high2float(m));
  const uint8_t scale = float_to_e4m3(inverse_scale * (amax * rcp_approx_ftz(6.0F)));
  const float block_scale = e4m3_to_float(scale);
  const float factor = block_scale == 0.0F ? 0.0F : rcp_approx_ftz(block_scale * rcp_approx_ftz(inverse_scale));
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float v[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(pairs[4 * h + i] << 16) * factor;
      v[2 * i + 1] = __uint_as_float(pairs[4 * h + i] & 0xFFFF0000u) * factor;
    }
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\tcvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\tcvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
        : "=r"(codes[h]) : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
  }
  return scale;
}

// Sixteen activations (eight BF16 pairs) as the kind's token values; `group`: number of the sixteen values inside the
// chunk.  Returns the FP4 block scale (0 otherwise).
template <StreamKind KIND>
__device__ __forceinline__ uint8_t put_tokens(uint8_t* chunk, uint32_t token, uint32_t group, const uint32_t* pairs, float inverse_scale,
                                              uint32_t* codes) {
  constexpr uint32_t kGroups = lane_values(KIND) / 16;
  const uint32_t lane = token % 8 * 4 + group / kGroups, j = group % kGroups;
  uint8_t scale = 0;
  if constexpr (KIND == StreamKind::w4a4) {
    scale = quantise_fp4(pairs, inverse_scale, codes);
    *reinterpret_cast<uint2*>(chunk + (j / 2) * 512 + lane * 16 + (j % 2) * 8) = make_uint2(codes[0], codes[1]);
    chunk[1024 + lane * 4 + j] = scale;
  } else if constexpr (KIND == StreamKind::w8a8) {        // e4m3_satfinite(x / input_scale), src/fp8_linear.cu:33-52
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      r[i] = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t w = pairs[2 * i + h];
        const uint32_t code = __nv_cvt_float2_to_fp8x2(
            make_float2(__fmul_rn(__uint_as_float(w << 16), inverse_scale), __fmul_rn(__uint_as_float(w & 0xFFFF0000u), inverse_scale)),
            __NV_SATFINITE, __NV_E4M3);
        r[i] |= code << (16 * h);
      }
    }
    *reinterpret_cast<uint4*>(chunk + j * 512 + lane * 16) = make_uint4(r[0], r[1], r[2], r[3]);
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t* p = pairs + 4 * h;
      uint4 r = make_uint4(p[0], p[1], p[2], p[3]);
      // values (0, 4), (1, 5), (2, 6), (3, 7), as the weights come
      if constexpr (KIND == StreamKind::w4a16)
        r = make_uint4(__byte_perm(p[0], p[2], 0x5410), __byte_perm(p[0], p[2], 0x7632), __byte_perm(p[1], p[3], 0x5410), __byte_perm(p[1], p[3], 0x7632));
      *reinterpret_cast<uint4*>(chunk + (2 * j + h) * 512 + lane * 16) = r;
    }
  }
  return scale;
}

// GeGLU of sixteen gate values (eight BF16 pairs, replaced) and the up values beside them.
__device__ __forceinline__ void geglu_pairs(const bf16* up, uint32_t* pairs) {
  const uint4 c = reinterpret_cast<const uint4*>(up)[0], d = reinterpret_cast<const uint4*>(up)[1];
  uint32_t u[8] = {c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
#pragma unroll 1
  for (int i = 0; i < 8; ++i) {
    const float lo = gelu_tanh_multiply_bf16(__uint_as_float(pairs[0] << 16), __uint_as_float(u[0] << 16));
    const float hi = gelu_tanh_multiply_bf16(__uint_as_float(pairs[0] & 0xFFFF0000u), __uint_as_float(u[0] & 0xFFFF0000u));
#pragma unroll
    for (int j = 0; j < 7; ++j) {                            // the next one comes to the front, the result goes to the end
      pairs[j] = pairs[j + 1];
      u[j] = u[j + 1];
    }
    pairs[7] = (__float_as_uint(lo) >> 16) | (__float_as_uint(hi) & 0xFFFF0000u);
  }
}

}  // namespace gw::stream
