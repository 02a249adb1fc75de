// The grouped GEMMs of MoE layers whose experts are all FP8 or all BF16 (or NVFP4 used as BF16 copies), on sm_100a: weights
// on the 128 lanes, an expert's token rows on the columns, as in gemm_moe_narrow.cu without block scales.
//
// What bounds them: the expert weights from HBM (761 MB in FP8, 1522 MB in BF16 when every expert has a row) as long as
// experts have a few dozen rows; then what a CTA takes in from L2 (16 KB of weights and up to 16 KB of tokens for four MMAs).
// The work is found from the expert offsets alone and the first ring of weights is asked for before the wait for the kernel
// in front.  Gate/up: a lane tile is 64 gate rows and the 64 up rows of the same channels (eleven tiles for 704 channels
// without padding), and the epilogue applies GeGLU and makes the input of the down GEMM, beside the BF16 intermediates that
// the workspace exposes.  Without scales there is nothing between a ring stage's arrival and its MMAs.
//
// Roles per CTA: warp 0 = producer (one lane), warp 1 = MMA issuer (one lane), the others = epilogue.  Every wait is bounded
// and reports through the device error word.  No load fans out to other CTAs.
#include <string>

#include "common.cuh"
#include "gemm_moe_plain.h"
#include "moe_work.cuh"
#include "pair.cuh"
#include "ptx.cuh"

namespace gw {
namespace {

using namespace moe_work;
using pair::report;

constexpr int kHidden = 2816;
constexpr int kInter = 704;
constexpr int kFirstEpilogueWarp = 2;
constexpr uint32_t kDescHiSw128 = uint32_t(1024 >> 4) | (1u << 14) | (2u << 29);   // SBO 1024 B, version 1, SWIZZLE_128B
constexpr int kMaxSmem = 227 * 1024;

__device__ __forceinline__ uint64_t make_desc(uint32_t lo16) { return (uint64_t(kDescHiSw128) << 32) | lo16; }

template <bool FP8, int TILE, bool FIRST>
struct Plain {
  static constexpr int kKBytes = (FIRST ? kHidden : kInter) * (FP8 ? 1 : 2);
  static constexpr int kKStages = (kKBytes + 127) / 128;            // ring stages of 128 bytes of K; the copy engine zero-fills the last
  static constexpr int kLastBlocks = (kKBytes - (kKStages - 1) * 128) / 32;   // MMAs of the last one
  static constexpr int kCTiles = FIRST ? kInter / 64 : kHidden / 128;
  static constexpr int kWgtBytes = 128 * 128, kTokBytes = TILE * 128, kStageBytes = kWgtBytes + kTokBytes;
  // gate/up: BF16 values of 64 tokens, transposed for the epilogue; 16 bytes against bank conflicts
  static constexpr int kPassTokens = 64, kPitch = 256 + 16;
  static constexpr int kFixedBytes = (FIRST ? kPassTokens * kPitch : 0) + 1024 + int(sizeof(WorkTable)) + 512;
  static constexpr int kStages = (kMaxSmem - kFixedBytes) / kStageBytes;
  static constexpr int kSmemBytes = kStages * kStageBytes + kFixedBytes;
  static constexpr int kTmemCols = 256;                              // two accumulators of up to 128 columns
  static constexpr int kEpilogueThreads = 32 * kEpilogueWarps<TILE>;
  static constexpr int kThreads = 32 * kFirstEpilogueWarp + kEpilogueThreads;
  static_assert((2 * kStages + 4) * 8 + 16 <= 512 - 16, "barriers");
  static_assert(kSmemBytes > 116 * 1024, "one CTA per SM is assumed by the tensor-memory allocation");
};

template <bool FP8, int TILE, bool FIRST>
__global__ void __launch_bounds__((Plain<FP8, TILE, FIRST>::kThreads), 1)
moe_plain_kernel(const __grid_constant__ PairMoeParams p) {
  using C = Plain<FP8, TILE, FIRST>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + C::kStages * C::kStageBytes;
  WorkTable* table = reinterpret_cast<WorkTable*>(staging + (FIRST ? C::kPassTokens * C::kPitch : 0));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(table) + (sizeof(WorkTable) + 15) / 16 * 16);
  uint64_t* empty_bar = full_bar + C::kStages;
  uint64_t* acc_full_bar = empty_bar + C::kStages;
  uint64_t* acc_empty_bar = acc_full_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) / 32, 0), lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      ptx::mbar_init(full_bar + s, 1);
      ptx::mbar_init(empty_bar + s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(acc_full_bar + a, 1);
      ptx::mbar_init(acc_empty_bar + a, kEpilogueWarps<TILE>);
    }
    *abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async_smem();
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, C::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // The kernel in front wrote the token rows; the offsets were written before it and the weights by no kernel of this call
  // (see common.cuh).  So the work is found and the first ring of weights is on its way before the wait.
  build_work_table<TILE, FIRST ? 0 : 2, FIRST ? 1 : 2>(p, table, C::kCTiles);
  if (warp != 0) griddep_enter();
  // CTAs take units in turn: the ones that run together are of the same few experts, whose token rows stay in L2 (one
  // contiguous range per CTA: BF16, 3000 tokens 805 us, so 568).
  const Range range{int(blockIdx.x), table->prefix[kExperts]};
  const int step = int(gridDim.x);
  const auto place = [&](int w, Unit& u) { return place_unit<TILE>(table, w, C::kCTiles, u); };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (one lane)
    if (ptx::elect_one()) {
      const uint64_t evict_first = ptx::l2_evict_first(), evict_normal = ptx::l2_evict_normal();
      int stage = 0;
      uint32_t phase = 0;
      Unit u{-1, 0, 0, 0, 0};
      bool waited = false;
      for (int w = range.begin; w < range.end && !*abort_flag; w += step) {
        const int tiles = place(w, u);
        const CUtensorMap* maps = p.map_table + u.e * kMoeMapsPerExpert;
        const uint64_t policy = tiles == 1 ? evict_first : evict_normal;     // weights that are read once leave L2 first
        const int token_row = u.first + u.tile * TILE;
        const auto weights = [&](int ks, int at) {
          uint8_t* base = smem + at * C::kStageBytes;
          ptx::mbar_expect_tx(full_bar + at, C::kStageBytes);
          if constexpr (FIRST) {
            ptx::tma_load_2d(base, maps + kMoeMapWideGate64, ks * 128, u.part * 64, full_bar + at, policy);
            ptx::tma_load_2d(base + C::kWgtBytes / 2, maps + kMoeMapWideUp64, ks * 128, u.part * 64, full_bar + at, policy);
          } else {
            ptx::tma_load_2d(base, maps + 6, ks * 128, u.part * 128, full_bar + at, policy);
          }
        };
        const auto tokens = [&](int ks, int at) {
          ptx::tma_load_2d(smem + at * C::kStageBytes + C::kWgtBytes, &p.map_tokens, ks * 128, token_row, full_bar + at);
        };
        int ks = 0;
        if (!waited) {
          constexpr int kAhead = C::kStages < C::kKStages ? C::kStages : C::kKStages;
          for (int i = 0; i < kAhead; ++i) weights(i, i);
          griddep_wait();
          waited = true;
          for (int i = 0; i < kAhead; ++i) tokens(i, i);
          ks = kAhead;
          if (kAhead < C::kStages) stage = kAhead; else phase = 1;
        }
        for (; ks < C::kKStages; ++ks) {
          if (!ptx::mbar_wait_bounded(empty_bar + stage, phase ^ 1)) {
            report(p.error, 0x1a000000u | (blockIdx.x << 8) | stage, abort_flag);
            break;
          }
          weights(ks, stage);
          tokens(ks, stage);
          if (++stage == C::kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (one lane)
    if (ptx::elect_one()) {
      int stage = 0, turn = 0;
      uint32_t phase = 0;
      Unit u{-1, 0, 0, 0, 0};
      const uint32_t smem_base16 = ptx::smem_u32(smem) >> 4;
      for (int w = range.begin; w < range.end && !*abort_flag; w += step, ++turn) {
        place(w, u);
        const int acc = turn & 1, columns = mma_columns(valid_columns(u, TILE));
        const uint32_t idesc = FP8 ? ptx::idesc_fp8(columns) : ptx::idesc_bf16(columns);
        if (!ptx::mbar_wait_bounded(acc_empty_bar + acc, (uint32_t(turn >> 1) & 1u) ^ 1u)) {
          report(p.error, 0x29000000u | (blockIdx.x << 8) | acc, abort_flag);
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t d = tmem_base + acc * TILE;
        bool failed = false;
        for (int ks = 0; ks < C::kKStages; ++ks) {
          if (!ptx::mbar_wait_bounded(full_bar + stage, phase)) {
            report(p.error, 0x39000000u | (blockIdx.x << 8) | stage, abort_flag);
            failed = true;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t base16 = smem_base16 + uint32_t(stage) * uint32_t(C::kStageBytes >> 4);
          const int blocks = ks + 1 == C::kKStages ? C::kLastBlocks : 4;
#pragma unroll
          for (int kb = 0; kb < 4; ++kb) {
            if (kb >= blocks) continue;
            const uint64_t a = make_desc(base16 + 2 * kb), b = make_desc(base16 + (C::kWgtBytes >> 4) + 2 * kb);
            if constexpr (FP8) ptx::tc_mma_fp8(d, a, b, idesc, (ks | kb) != 0 ? 1u : 0u);
            else ptx::tc_mma_bf16(d, a, b, idesc, (ks | kb) != 0 ? 1u : 0u);
          }
          ptx::tc_commit(empty_bar + stage);
          if (++stage == C::kStages) { stage = 0; phase ^= 1; }
        }
        if (failed) break;
        ptx::tc_commit(acc_full_bar + acc);
      }
    }
    __syncwarp();
  } else {
    const int quad = warp % 4, which = (warp - kFirstEpilogueWarp) / 4;      // lanes; every second or fourth chunk of 16 tokens
    int turn = 0;
    Unit u{-1, 0, 0, 0, 0};
    for (int w = range.begin; w < range.end; w += step, ++turn) {
      place(w, u);
      const int acc = turn & 1;
      const int valid = valid_columns(u, TILE);
      // this lane's multiplier; BF16 has none (an expert's alpha belongs to its NVFP4 form)
      float alpha = 1.0F;
      if constexpr (FP8) {
        const int proj = FIRST ? quad / 2 : 2, channel = FIRST ? u.part * 64 + quad % 2 * 32 + lane : u.part * 128 + quad * 32 + lane;
        const float* per_channel = p.experts[u.e].channel_alpha[proj];
        alpha = per_channel != nullptr ? per_channel[channel] : p.experts[u.e].alpha[proj];
      }
      const bool arrived = ptx::mbar_wait_warp(acc_full_bar + acc, uint32_t(turn >> 1) & 1u);
      if (!arrived) report(p.error, 0x48000000u | (blockIdx.x << 8) | acc, abort_flag);
      if constexpr (FIRST) {
        if (epilogue_barrier_any<C::kEpilogueThreads>(!arrived)) break;      // and the staging buffer is free again
      } else {
        if (!arrived) break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + acc * TILE + (uint32_t(quad * 32) << 16);
      if constexpr (FIRST) {
        // ---------------------------------------------------------------- gate/up: GeGLU and the input of the down GEMM
        // As in gemm_moe_narrow.cu: through shared memory as [token][gate 64 | up 64], then eight channels of a token a thread.
        const int tid = int(threadIdx.x) - 32 * kFirstEpilogueWarp;
        const int channels = tid % 8 * 8;
        const float inverse_scale = p.experts[u.e].inverse_input_scale[2];
#pragma unroll 1
        for (int pass = 0; pass < valid; pass += C::kPassTokens) {
          const int in_pass = min(C::kPassTokens, valid - pass);
          uint16_t* mine = reinterpret_cast<uint16_t*>(staging) + quad * 32 + lane;
#pragma unroll 1
          for (int c0 = which * 16; c0 < in_pass; c0 += kEpilogueWarps<TILE> * 4) {
            uint32_t r[16];
            ptx::tmem_load16(taddr + pass + c0, r);
            ptx::tmem_load_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const bf16 v = __float2bfloat16_rn(__fmul_rn(__uint_as_float(r[i]), alpha));
              mine[(c0 + i) * (C::kPitch / 2)] = *reinterpret_cast<const uint16_t*>(&v);
            }
          }
          if (pass + C::kPassTokens >= valid) {
            ptx::tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(acc_empty_bar + acc);            // the tile after next may start
          }
          epilogue_barrier<C::kEpilogueThreads>();
#pragma unroll 1
          for (int token = tid / 8; token < in_pass; token += C::kEpilogueThreads / 8) {
            const uint32_t from = ptx::smem_u32(staging) + uint32_t(token) * C::kPitch + channels * 2;
            const uint4 g = ptx::lds128(from), v = ptx::lds128(from + 128);
            const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {v.x, v.y, v.z, v.w};
            uint32_t aw[4], codes[2] = {0, 0};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float lo = gelu_tanh_multiply_bf16(__uint_as_float(gw[i] << 16), __uint_as_float(uw[i] << 16));
              const float hi = gelu_tanh_multiply_bf16(__uint_as_float(gw[i] & 0xFFFF0000u), __uint_as_float(uw[i] & 0xFFFF0000u));
              aw[i] = (__float_as_uint(lo) >> 16) | (__float_as_uint(hi) & 0xFFFF0000u);
              if constexpr (FP8)
                codes[i / 2] |= (uint32_t(float_to_e4m3(__fmul_rn(lo, inverse_scale))) | uint32_t(float_to_e4m3(__fmul_rn(hi, inverse_scale))) << 8)
                                << (16 * (i % 2));
            }
            const size_t row = size_t(u.first) + u.tile * TILE + pass + token;
            const int channel = u.part * 64 + channels;
            bf16* gate_up = static_cast<bf16*>(p.capture_gate_up) + row * (2 * size_t(kInter)) + channel;
            *reinterpret_cast<uint4*>(gate_up) = g;
            *reinterpret_cast<uint4*>(gate_up + kInter) = v;
            *reinterpret_cast<uint4*>(static_cast<bf16*>(p.capture_activated) + row * size_t(kInter) + channel) = make_uint4(aw[0], aw[1], aw[2], aw[3]);
            if constexpr (FP8) *reinterpret_cast<uint2*>(p.packed_out + row * size_t(kInter) + channel) = make_uint2(codes[0], codes[1]);
          }
          if (C::kPassTokens < TILE && pass + C::kPassTokens < valid) epilogue_barrier<C::kEpilogueThreads>();     // the staging buffer is free again
        }
      } else {
        // ---------------------------------------------------------------- down: BF16 rows, 64 contiguous bytes of a token a warp
        bf16* out = static_cast<bf16*>(p.out) + (size_t(u.first) + u.tile * TILE) * size_t(kHidden) + u.part * 128 + quad * 32 + lane;
#pragma unroll 1
        for (int c0 = which * 16; c0 < valid; c0 += kEpilogueWarps<TILE> * 4) {
          uint32_t r[16];
          ptx::tmem_load16(taddr + c0, r);
          ptx::tmem_load_wait();
          bf16* dst = out + c0 * size_t(kHidden);
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (c0 + i < valid) dst[i * kHidden] = __float2bfloat16_rn(__fmul_rn(__uint_as_float(r[i]), alpha));
        }
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(acc_empty_bar + acc);
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <bool FP8, int TILE, bool FIRST>
cudaError_t launch_instance(const PairMoeParams& params, int sm_count, cudaStream_t stream) {
  using C = Plain<FP8, TILE, FIRST>;
  static bool configured_on[kMaxDeviceSlots] = {};   // the attribute is per GPU
  bool& configured = configured_on[current_device_slot()];
  if (!configured) {
    const cudaError_t status = cudaFuncSetAttribute(moe_plain_kernel<FP8, TILE, FIRST>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
    if (status != cudaSuccess) return status;
    configured = true;
  }
  return launch_pdl_shared(moe_plain_kernel<FP8, TILE, FIRST>, dim3(sm_count), dim3(C::kThreads), size_t(C::kSmemBytes), stream, params);
}

template <bool FIRST>
cudaError_t launch_stage(int tile_rows, const PairMoeParams& params, int sm_count, cudaStream_t stream) {
  const bool fp8 = params.kind == kMoeKindFp8;
  if (tile_rows == 64) return fp8 ? launch_instance<true, 64, FIRST>(params, sm_count, stream) : launch_instance<false, 64, FIRST>(params, sm_count, stream);
  if (tile_rows == 128) return fp8 ? launch_instance<true, 128, FIRST>(params, sm_count, stream) : launch_instance<false, 128, FIRST>(params, sm_count, stream);
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_moe_plain_gate_up(int tile_rows, const PairMoeParams& params, int sm_count, cudaStream_t stream) {
  return launch_stage<true>(tile_rows, params, sm_count, stream);
}
cudaError_t launch_moe_plain_down(int tile_rows, const PairMoeParams& params, int sm_count, cudaStream_t stream) {
  return launch_stage<false>(tile_rows, params, sm_count, stream);
}

}  // namespace gw
