// The two grouped NVFP4 GEMMs of the MoE layer for batches whose experts get a few dozen rows each (tcgen05, one CTA
// per tile), on sm_100a: weights on the 128 lanes, an expert's token rows on the columns (moe.cu:489-534 of the
// reference runs CUTLASS grouped GEMMs, moe_nvfp4.cuh:15-132).
//
// What bounds them: the expert weights from HBM (428 MB when every expert has a row).  So
//   - nothing but the expert offsets is read to find the work (moe_work.cuh): no descriptor launch in front, and none of
//     its 152 bytes to fetch for a tile;
//   - gate/up: a lane tile is 64 gate rows and the 64 up rows of the same channels, eleven tiles for 704 channels without
//     padding, and the epilogue applies GeGLU and quantises the down input: no BF16 intermediate has to travel and no
//     launch stands between the two GEMMs;
//   - down: the token rows stay in shared memory while the CTA sweeps the output channels; the MMA lane waits for the
//     weight slabs themselves, the scales of a whole unit (K = 704) go to tensor memory in one round.
// A CTA walks one contiguous range of units, so it changes experts once or twice, and asks for its first ring of weights
// before it waits for the kernel in front.
//
// Measured (whole MoE layer, us, these kernels / group descriptors + gemm_tc.cu + a GeGLU kernel up to 512 tokens and the
// CTA-pair kernels beyond): 4 tokens 35 / 48, 64 81 / 104, 256 104 / 127, 777 115 / 157, 2048 178 / 186; with popular experts
// (1.2 power law) 64 45 / 63, 256 75 / 102, 777 105 / 133, 2048 176 / 197.  64 tokens: gate/up 40 us for 281 MB of weights.
//
// Roles per CTA, as in gemm_tc.cu: warp 0 = producer (one lane), warp 1 = MMA issuer (one lane), warps 2..5 = scale
// loaders (shared memory -> registers -> tensor memory), warps 6 and up = epilogue.  Every wait is bounded and reports
// through the device error word.  No load fans out to other CTAs.
#include <string>

#include "common.cuh"
#include "gemm_moe_narrow.h"
#include "moe_work.cuh"
#include "pair.cuh"
#include "ptx.cuh"

namespace gw {
namespace {

using namespace moe_work;
using pair::report;

constexpr int kHidden = 2816;
constexpr int kInter = 704;
constexpr int kScaleWarps = 4, kFirstEpilogueWarp = 2 + kScaleWarps;
template <int TILE> constexpr int kThreads = 32 * (kFirstEpilogueWarp + kEpilogueWarps<TILE>);
constexpr int kTmemCols = 512;
constexpr uint32_t kDescHiSw128 = uint32_t(1024 >> 4) | (1u << 14) | (2u << 29);   // SBO 1024 B, version 1, SWIZZLE_128B
constexpr int kMaxSmem = 227 * 1024;

__device__ __forceinline__ uint64_t make_desc(uint32_t lo16) { return (uint64_t(kDescHiSw128) << 32) | lo16; }

__device__ __forceinline__ uint2 lds64(uint32_t address) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(address));
  return v;
}
// The four 32-row words of a lane in a 128-row scale atom, so that the tile's first 32-row group comes first.
__device__ __forceinline__ uint4 rotated(uint4 v, uint32_t sub) {
  if (sub & 1) v = make_uint4(v.y, v.z, v.w, v.x);
  if (sub & 2) v = make_uint4(v.z, v.w, v.x, v.y);
  return v;
}

// ===========================================================================
// gate/up: Y = Xq . [Wgate | Wup]^T per expert, GeGLU, FP4 quantisation of the result
// ===========================================================================
template <int TILE>
struct GateUp {
  static constexpr int kEpilogueThreads = 32 * kEpilogueWarps<TILE>;
  static constexpr int kKBlocks = 4;                       // MMAs (K = 64 each) per stage
  static constexpr int kKStages = kHidden / 2 / 128;       // 11 stages of 128 bytes of K
  static constexpr int kKAtoms = kHidden / 64;             // 44 scale atoms per 128-row block
  static constexpr int kCTiles = kInter / 64;              // 11 channel tiles
  static constexpr int kWgtBytes = 128 * 128;              // 64 gate rows, then 64 up rows, x 128 bytes of K
  static constexpr int kTokBytes = TILE * 128;
  static constexpr int kAtomsBytes = kKBlocks * 512;       // four scale atoms: of the tokens, of gate, of up
  static constexpr int kStageBytes = kWgtBytes + kTokBytes + 3 * kAtomsBytes;
  // BF16 gate and up values of up to 64 tokens, transposed for the epilogue: 128 values a token and 16 bytes against
  // bank conflicts
  static constexpr int kPassTokens = 64;
  static constexpr int kPitch = 256 + 16;
  static constexpr int kFixedBytes = kPassTokens * kPitch + 1024 + int(sizeof(WorkTable)) + 512;
  static constexpr int kStagesRaw = (kMaxSmem - kFixedBytes) / kStageBytes;
  static constexpr int kStages = kStagesRaw < 8 ? kStagesRaw : 8;
  static constexpr int kSmemBytes = kStages * kStageBytes + kFixedBytes;
  static constexpr int kAccCols = 2 * TILE;
  static constexpr int kSfSlotCols = kKBlocks * 8;         // weights 4 columns and tokens 4 columns per K block
  static_assert(kAccCols + kStages * kSfSlotCols <= kTmemCols, "tensor memory over-subscribed");
  static_assert((4 * kStages + 4) * 8 + 16 <= 512, "barriers");
  static_assert(kSmemBytes > 116 * 1024, "one CTA per SM is assumed by the tensor-memory allocation");
};

template <int TILE>
__global__ void __launch_bounds__(kThreads<TILE>, 1)
moe_narrow_gate_up_kernel(const __grid_constant__ PairMoeParams p) {
  using C = GateUp<TILE>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + C::kStages * C::kStageBytes;
  WorkTable* table = reinterpret_cast<WorkTable*>(staging + C::kPassTokens * C::kPitch);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(table) + (sizeof(WorkTable) + 15) / 16 * 16);
  uint64_t* sf_full_bar = full_bar + C::kStages;
  uint64_t* sf_ready_bar = sf_full_bar + C::kStages;
  uint64_t* empty_bar = sf_ready_bar + C::kStages;
  uint64_t* acc_full_bar = empty_bar + C::kStages;
  uint64_t* acc_empty_bar = acc_full_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) / 32, 0), lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kStages; ++s) {
      ptx::mbar_init(full_bar + s, 1);
      ptx::mbar_init(sf_full_bar + s, 1);
      ptx::mbar_init(sf_ready_bar + s, kScaleWarps);
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
    ptx::tmem_alloc(tmem_slot, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // The kernel in front quantised the rows; the offsets were written before it and the weights by no kernel of this call
  // (see common.cuh).  So the work is found and the first ring of weights is on its way before the wait.
  build_work_table<TILE, 0, 1>(p, table, C::kCTiles);
  if (warp != 0) griddep_enter();
  const Range range = my_range(table->prefix[kExperts]);
  const auto place = [&](int w, Unit& u) { return place_unit<TILE>(table, w, C::kCTiles, u); };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (one lane)
    if (ptx::elect_one()) {
      const uint64_t evict_first = ptx::l2_evict_first(), evict_normal = ptx::l2_evict_normal();
      int stage = 0;
      uint32_t phase = 0;
      Unit u{-1, 0, 0, 0, 0};
      const uint8_t *sf_gate = nullptr, *sf_up = nullptr;
      int info_of = -1;
      bool waited = false;
      for (int w = range.begin; w < range.end && !*abort_flag; ++w) {
        const int tiles = place(w, u);
        if (info_of != u.e) {
          sf_gate = p.experts[u.e].scales[0];
          sf_up = p.experts[u.e].scales[1];
          info_of = u.e;
        }
        const CUtensorMap* map_gate = p.map_table + u.e * kMoeMapsPerExpert + kMoeMapGate64;
        const CUtensorMap* map_up = p.map_table + u.e * kMoeMapsPerExpert + kMoeMapUp64;
        const uint64_t policy = tiles == 1 ? evict_first : evict_normal;     // weights that are read once leave L2 first
        const int token_row = u.first + u.tile * TILE;
        const uint8_t* sft = p.sf_tokens + (size_t(u.first / 128 + u.e) + u.tile * TILE / 128) * size_t(C::kKAtoms) * 512;
        const size_t sfw = size_t(u.part / 2) * C::kKAtoms * 512;
        const auto weights = [&](int ks, int at_stage) {
          uint8_t* base = smem + at_stage * C::kStageBytes;
          uint8_t* atoms = base + C::kWgtBytes + C::kTokBytes;
          uint64_t *bar = full_bar + at_stage, *sf_bar = sf_full_bar + at_stage;
          const size_t at = sfw + size_t(ks) * C::kAtomsBytes;
          ptx::mbar_expect_tx(bar, C::kWgtBytes + C::kTokBytes);
          ptx::tma_load_2d(base, map_gate, ks * 128, u.part * 64, bar, policy);
          ptx::tma_load_2d(base + C::kWgtBytes / 2, map_up, ks * 128, u.part * 64, bar, policy);
          ptx::mbar_expect_tx(sf_bar, 3 * C::kAtomsBytes);
          ptx::bulk_load(atoms + C::kAtomsBytes, sf_gate + at, C::kAtomsBytes, sf_bar);
          ptx::bulk_load(atoms + 2 * C::kAtomsBytes, sf_up + at, C::kAtomsBytes, sf_bar);
        };
        const auto tokens = [&](int ks, int at_stage) {
          uint8_t* base = smem + at_stage * C::kStageBytes;
          ptx::bulk_load(base + C::kWgtBytes + C::kTokBytes, sft + size_t(ks) * C::kAtomsBytes, C::kAtomsBytes, sf_full_bar + at_stage);
          ptx::tma_load_2d(base + C::kWgtBytes, &p.map_tokens, ks * 128, token_row, full_bar + at_stage);
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
            report(p.error, 0x16000000u | (blockIdx.x << 8) | stage, abort_flag);
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
      for (int w = range.begin; w < range.end && !*abort_flag; ++w, ++turn) {
        place(w, u);
        const int acc = turn & 1;
        const uint32_t idesc = ptx::idesc_nvfp4(mma_columns(valid_columns(u, TILE)));
        if (!ptx::mbar_wait_bounded(acc_empty_bar + acc, (uint32_t(turn >> 1) & 1u) ^ 1u)) {
          report(p.error, 0x26000000u | (blockIdx.x << 8) | acc, abort_flag);
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t d = tmem_base + acc * TILE;
        bool failed = false;
        for (int ks = 0; ks < C::kKStages; ++ks) {
          // the loader warps arrive after the stage's operands have landed too
          if (!ptx::mbar_wait_bounded(sf_ready_bar + stage, phase)) {
            report(p.error, 0x36000000u | (blockIdx.x << 8) | stage, abort_flag);
            failed = true;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t base16 = smem_base16 + uint32_t(stage) * uint32_t(C::kStageBytes >> 4);
          const uint32_t sf = tmem_base + C::kAccCols + uint32_t(stage) * C::kSfSlotCols;
#pragma unroll
          for (int kb = 0; kb < C::kKBlocks; ++kb)
            ptx::tc_mma_nvfp4(d, make_desc(base16 + 2 * kb), make_desc(base16 + (C::kWgtBytes >> 4) + 2 * kb), idesc, sf + 4 * kb,
                              sf + 4 * C::kKBlocks + 4 * kb, (ks | kb) != 0 ? 1u : 0u);
          ptx::tc_commit(empty_bar + stage);
          if (++stage == C::kStages) { stage = 0; phase ^= 1; }
        }
        if (failed) break;
        ptx::tc_commit(acc_full_bar + acc);
      }
    }
    __syncwarp();
  } else if (warp < kFirstEpilogueWarp) {
    // ------------------------------------------------------------------ scale loaders
    // Lane r of an atom has the scales of the rows r, r + 32, r + 64, r + 96 of a 128-row block.  The weight tile's rows are
    // one half of a block of gate and of up: two words of each are the tile's four 32-row groups.
    const uint32_t quad_lane = uint32_t((warp % 4) * 32) << 16;
    int stage = 0;
    uint32_t phase = 0;
    Unit u{-1, 0, 0, 0, 0};
    for (int w = range.begin; w < range.end && !*abort_flag; ++w) {
      place(w, u);
      const uint32_t sub = TILE < 128 ? uint32_t(u.tile * TILE % 128) / 32 : 0;
      const uint32_t half = uint32_t(u.part & 1) * 8;
      bool failed = false;
      for (int ks = 0; ks < C::kKStages; ++ks) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(sf_full_bar + stage, phase))) {
          report(p.error, 0x68000000u | (blockIdx.x << 8) | stage, abort_flag);
          failed = true;
          break;
        }
        const uint32_t src = ptx::smem_u32(smem + stage * C::kStageBytes + C::kWgtBytes + C::kTokBytes) + lane * 16;
        const uint32_t slot = tmem_base + C::kAccCols + uint32_t(stage) * C::kSfSlotCols + quad_lane;
        uint32_t r[16], t[16];
#pragma unroll
        for (int kb = 0; kb < C::kKBlocks; ++kb) {
          const uint2 g = lds64(src + C::kAtomsBytes + kb * 512 + half), v = lds64(src + 2 * C::kAtomsBytes + kb * 512 + half);
          r[4 * kb] = g.x; r[4 * kb + 1] = g.y; r[4 * kb + 2] = v.x; r[4 * kb + 3] = v.y;
          const uint4 x = rotated(ptx::lds128(src + kb * 512), sub);
          t[4 * kb] = x.x; t[4 * kb + 1] = x.y; t[4 * kb + 2] = x.z; t[4 * kb + 3] = x.w;
        }
        ptx::tmem_store16(slot, r);
        ptx::tmem_store16(slot + 4 * C::kKBlocks, t);
        ptx::tmem_store_wait();
        ptx::tc_fence_before_sync();
        // the arrival also vouches for the operand tiles
        if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(full_bar + stage, phase))) {
          report(p.error, 0x69000000u | (blockIdx.x << 8) | stage, abort_flag);
          failed = true;
          break;
        }
        if (lane == 0) ptx::mbar_arrive(sf_ready_bar + stage);
        if (++stage == C::kStages) { stage = 0; phase ^= 1; }
      }
      if (failed) break;
    }
  } else {
    // ------------------------------------------------------------------ epilogue: GeGLU + FP4 quantise
    // The gate lanes (0..63) and the up lanes (64..127) of a channel belong to different warps: the scaled accumulators,
    // rounded to BF16, which is what GeGLU consumes, go through shared memory as [token][gate 64 | up 64].  Then eight
    // threads share a token's 64 channels, eight channels each: 32 contiguous bytes of codes, four scale bytes.
    const int quad = warp % 4, which = (warp - kFirstEpilogueWarp) / 4;      // lanes; every second or fourth chunk of 16 tokens
    const int tid = int(threadIdx.x) - 32 * kFirstEpilogueWarp;
    const int channels = tid % 8 * 8;                                        // this thread's eight of the tile's 64 channels
    Unit u{-1, 0, 0, 0, 0};
    float alpha = 0.0F, inverse_scale = 0.0F;
    int info_of = -1, turn = 0;
    bf16* cap_gu = static_cast<bf16*>(p.capture_gate_up);
    bf16* cap_act = static_cast<bf16*>(p.capture_activated);
    for (int w = range.begin; w < range.end; ++w, ++turn) {
      place(w, u);
      if (info_of != u.e) {
        alpha = p.experts[u.e].alpha[quad < 2 ? 0 : 1];
        inverse_scale = p.experts[u.e].inverse_input_scale[2];
        info_of = u.e;
      }
      const int acc = turn & 1;
      const int valid = valid_columns(u, TILE);
      const bool arrived = ptx::mbar_wait_warp(acc_full_bar + acc, uint32_t(turn >> 1) & 1u);
      if (!arrived) report(p.error, 0x46000000u | (blockIdx.x << 8) | acc, abort_flag);
      if (epilogue_barrier_any<C::kEpilogueThreads>(!arrived)) break;                             // and the staging buffer is free again
      ptx::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + acc * TILE + (uint32_t(quad * 32) << 16);
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
          if (lane == 0) ptx::mbar_arrive(acc_empty_bar + acc);              // the tile after next may start
        }
        epilogue_barrier<C::kEpilogueThreads>();
#pragma unroll 1
        for (int base = 0; base < in_pass; base += C::kEpilogueThreads / 8) {
          const int token = base + tid / 8;
          const bool live = token < in_pass;                                 // the eight threads of a token agree
          const uint32_t from = ptx::smem_u32(staging) + uint32_t(live ? token : 0) * C::kPitch + channels * 2;
          const uint4 g = ptx::lds128(from), v = ptx::lds128(from + 128);
          const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {v.x, v.y, v.z, v.w};
          float act[8], amax = 0.0F;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            act[2 * i] = gelu_tanh_multiply_bf16(__uint_as_float(gw[i] << 16), __uint_as_float(uw[i] << 16));
            act[2 * i + 1] = gelu_tanh_multiply_bf16(__uint_as_float(gw[i] & 0xFFFF0000u), __uint_as_float(uw[i] & 0xFFFF0000u));
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(act[i]));
          amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));         // a K16 block is two threads'
          const uint8_t code = float_to_e4m3(inverse_scale * (amax * rcp_approx_ftz(6.0F)));
          const float block_scale = e4m3_to_float(code);
          const float factor = block_scale == 0.0F ? 0.0F : rcp_approx_ftz(block_scale * rcp_approx_ftz(inverse_scale));
          uint32_t packed = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) packed |= uint32_t(float2_to_e2m1x2(act[2 * i] * factor, act[2 * i + 1] * factor)) << (8 * i);
          uint32_t scales = code;                                            // the first thread gathers the token's four
          scales |= __shfl_down_sync(0xffffffffu, scales, 2) << 8;
          scales |= __shfl_down_sync(0xffffffffu, scales, 4) << 16;
          if (live) {
            const int l_index = u.tile * TILE + pass + token;                // row inside the expert
            const size_t row = size_t(u.first) + l_index;
            const int channel = u.part * 64 + channels;
            if (cap_gu != nullptr) {
              uint32_t aw[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) aw[i] = (__float_as_uint(act[2 * i]) >> 16) | (__float_as_uint(act[2 * i + 1]) & 0xFFFF0000u);
              *reinterpret_cast<uint4*>(cap_gu + row * (2 * size_t(kInter)) + channel) = g;
              *reinterpret_cast<uint4*>(cap_gu + row * (2 * size_t(kInter)) + kInter + channel) = v;
              *reinterpret_cast<uint4*>(cap_act + row * size_t(kInter) + channel) = make_uint4(aw[0], aw[1], aw[2], aw[3]);
            }
            if (p.records_out != nullptr) {
              uint8_t* record = p.records_out + row * size_t(kEpActivationRecordBytes);
              *reinterpret_cast<uint32_t*>(record + channel / 2) = packed;
              if (tid % 8 == 0) *reinterpret_cast<uint32_t*>(record + kInter / 2 + channel / 16) = scales;
            } else {
              *reinterpret_cast<uint32_t*>(p.packed_out + row * size_t(kInter / 2) + channel / 2) = packed;
              const size_t region = size_t(u.first / 128 + u.e) * 128 * (kInter / 16);
              if (tid % 8 == 0) *reinterpret_cast<uint32_t*>(p.scales_out + region + scale_offset(l_index, channel / 16, kInter)) = scales;
            }
          }
        }
        if (C::kPassTokens < TILE && pass + C::kPassTokens < valid) epilogue_barrier<C::kEpilogueThreads>();     // the staging buffer is free again
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ===========================================================================
// down: Y = Aq . Wdown^T per expert, BF16 rows out
// ===========================================================================
template <int TILE>
struct Down {
  static constexpr int kSlabs = 3;                         // 128 bytes of K each, the last one zero-filled past byte 352
  static constexpr int kKBlocks = kInter / 64;             // 11 MMAs (K = 64)
  static constexpr int kSfBytes = kKBlocks * 512;          // the 11 scale atoms of a 128-row block
  static constexpr int kSfRoom = 12 * 512;                 // copied to tensor memory 16 columns (4 atoms) at a time
  static constexpr int kWgtSlab = 128 * 128, kTokSlab = TILE * 128;
  static constexpr int kTokBytes = kSlabs * kTokSlab + kSfRoom;
  static constexpr int kBuffers = 2;                       // the next expert's rows arrive while this one's are in use
  static constexpr int kSfSlots = 3;                       // units whose weight scales are here
  static constexpr int kCTiles = kHidden / 128;            // 22
  static constexpr int kFixedBytes = kBuffers * kTokBytes + kSfSlots * kSfRoom + 1024 + int(sizeof(WorkTable)) + 512;
  static constexpr int kRing = (kMaxSmem - kFixedBytes) / kWgtSlab;        // weight slabs
  static constexpr int kSmemBytes = kRing * kWgtSlab + kFixedBytes;
  static constexpr int kAccCols = 2 * TILE;
  static constexpr int kSfSlotCols = 48;                   // 12 atoms x 4 columns
  static constexpr int kSfTokCol = kAccCols;               // + buffer * kSfSlotCols
  static constexpr int kSfWgtCol = kSfTokCol + kBuffers * kSfSlotCols;     // + slot * kSfSlotCols
  static_assert(kSfWgtCol + kSfSlots * kSfSlotCols <= kTmemCols, "tensor memory over-subscribed");
  static_assert(kSmemBytes <= kMaxSmem && kRing >= 2 * kSlabs, "shared memory over-subscribed");
  static_assert(kSmemBytes > 116 * 1024, "one CTA per SM is assumed by the tensor-memory allocation");
  static_assert((2 * kRing + 3 * kSfSlots + 3 * kBuffers + 4) * 8 + 16 <= 512 - 16, "barriers");
};

template <int TILE>
__global__ void __launch_bounds__(kThreads<TILE>, 1)
moe_narrow_down_kernel(const __grid_constant__ PairMoeParams p) {
  using C = Down<TILE>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* token_buf = smem + C::kRing * C::kWgtSlab;
  uint8_t* sf_buf = token_buf + C::kBuffers * C::kTokBytes;
  WorkTable* table = reinterpret_cast<WorkTable*>(sf_buf + C::kSfSlots * C::kSfRoom);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(table) + (sizeof(WorkTable) + 15) / 16 * 16);
  uint64_t* empty_bar = full_bar + C::kRing;
  uint64_t* sf_full_bar = empty_bar + C::kRing;
  uint64_t* sf_ready_bar = sf_full_bar + C::kSfSlots;
  uint64_t* sf_empty_bar = sf_ready_bar + C::kSfSlots;
  uint64_t* tok_full_bar = sf_empty_bar + C::kSfSlots;
  uint64_t* tok_ready_bar = tok_full_bar + C::kBuffers;
  uint64_t* tok_empty_bar = tok_ready_bar + C::kBuffers;
  uint64_t* acc_full_bar = tok_empty_bar + C::kBuffers;
  uint64_t* acc_empty_bar = acc_full_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) / 32, 0), lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kRing; ++s) {
      ptx::mbar_init(full_bar + s, 1);
      ptx::mbar_init(empty_bar + s, 1);
    }
    for (int s = 0; s < C::kSfSlots; ++s) {
      ptx::mbar_init(sf_full_bar + s, 1);
      ptx::mbar_init(sf_ready_bar + s, kScaleWarps);
      ptx::mbar_init(sf_empty_bar + s, 1);
    }
    for (int b = 0; b < C::kBuffers; ++b) {
      ptx::mbar_init(tok_full_bar + b, 1);
      ptx::mbar_init(tok_ready_bar + b, kScaleWarps);
      ptx::mbar_init(tok_empty_bar + b, 1);
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
    ptx::tmem_alloc(tmem_slot, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  build_work_table<TILE, 2, 2>(p, table, C::kCTiles);       // before the wait, as above
  if (warp != 0) griddep_enter();
  const Range range = my_range(table->prefix[kExperts]);
  // A ring position and the parity of its turn.
  struct Cursor {
    int at = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void step(int size) { if (++at == size) { at = 0; phase ^= 1; } }
  };
  // Token rows: `group` counts the changes of expert or token tile.
  struct Rows {
    int group = -1, tile_of = -1, expert_of = -1;
    __device__ __forceinline__ bool changed(const Unit& u) {
      if (expert_of == u.e && tile_of == u.tile) return false;
      expert_of = u.e;
      tile_of = u.tile;
      ++group;
      return true;
    }
    __device__ __forceinline__ int buffer() const { return group % C::kBuffers; }
    __device__ __forceinline__ uint32_t phase() const { return uint32_t(group / C::kBuffers) & 1u; }
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (one lane)
    if (ptx::elect_one()) {
      const uint64_t evict_first = ptx::l2_evict_first(), evict_normal = ptx::l2_evict_normal();
      Cursor slab, slot;
      Rows rows;
      Unit u{-1, 0, 0, 0, 0};
      bool failed = false;
      const auto weights = [&]() {
        if (!ptx::mbar_wait_bounded(sf_empty_bar + slot.at, slot.phase ^ 1)) {
          report(p.error, 0x17000000u | (blockIdx.x << 8) | slot.at, abort_flag);
          return false;
        }
        ptx::mbar_expect_tx(sf_full_bar + slot.at, C::kSfBytes);
        ptx::bulk_load(sf_buf + slot.at * C::kSfRoom, p.experts[u.e].scales[2] + size_t(u.part) * C::kSfBytes, C::kSfBytes, sf_full_bar + slot.at);
        slot.step(C::kSfSlots);
        const CUtensorMap* map_weights = p.map_table + u.e * kMoeMapsPerExpert + 2;
        const uint64_t policy = u.count <= TILE ? evict_first : evict_normal;     // weights that are read once leave L2 first
        for (int j = 0; j < C::kSlabs; ++j) {
          if (!ptx::mbar_wait_bounded(empty_bar + slab.at, slab.phase ^ 1)) {
            report(p.error, 0x18000000u | (blockIdx.x << 8) | slab.at, abort_flag);
            return false;
          }
          ptx::mbar_expect_tx(full_bar + slab.at, C::kWgtSlab);
          ptx::tma_load_2d(smem + slab.at * C::kWgtSlab, map_weights, j * 128, u.part * 128, full_bar + slab.at, policy);
          slab.step(C::kRing);
        }
        return true;
      };
      constexpr int kFit = C::kRing / C::kSlabs < C::kSfSlots ? C::kRing / C::kSlabs : C::kSfSlots;
      const int ahead = min(kFit, range.end - range.begin);
      for (int i = 0; i < ahead; ++i) {
        decode_unit(table, range.begin + i, C::kCTiles, u);
        weights();                                                  // every barrier is free: no wait
      }
      griddep_wait();
      for (int w = range.begin; w < range.end && !failed && !*abort_flag; ++w) {
        decode_unit(table, w, C::kCTiles, u);
        if (rows.changed(u)) {
          const int buffer = rows.buffer();
          if (!ptx::mbar_wait_bounded(tok_empty_bar + buffer, rows.phase() ^ 1)) {
            report(p.error, 0x19000000u | (blockIdx.x << 8) | buffer, abort_flag);
            break;
          }
          uint8_t* to = token_buf + buffer * C::kTokBytes;
          uint64_t* tok_bar = tok_full_bar + buffer;
          ptx::mbar_expect_tx(tok_bar, C::kSlabs * C::kTokSlab + C::kSfBytes);
          ptx::bulk_load(to + C::kSlabs * C::kTokSlab,
                         p.sf_tokens + (size_t(u.first / 128 + u.e) + u.tile * TILE / 128) * size_t(C::kSfBytes), C::kSfBytes, tok_bar);
#pragma unroll
          for (int j = 0; j < C::kSlabs; ++j)
            ptx::tma_load_2d(to + j * C::kTokSlab, &p.map_tokens, j * 128, u.first + u.tile * TILE, tok_bar);
        }
        if (w - range.begin >= ahead) failed = !weights();
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (one lane)
    if (ptx::elect_one()) {
      Cursor slab, slot;
      Rows rows;
      int turn = 0;
      Unit u{-1, 0, 0, 0, 0};
      bool failed = false;
      const uint32_t smem_base16 = ptx::smem_u32(smem) >> 4, tok_base16 = ptx::smem_u32(token_buf) >> 4;
      for (int w = range.begin; w < range.end && !failed && !*abort_flag; ++w, ++turn) {
        decode_unit(table, w, C::kCTiles, u);
        const int before = rows.group;
        if (rows.changed(u)) {
          if (before >= 0) ptx::tc_commit(tok_empty_bar + before % C::kBuffers);
          if (!ptx::mbar_wait_bounded(tok_ready_bar + rows.buffer(), rows.phase())) {
            report(p.error, 0x27000000u | (blockIdx.x << 8) | rows.buffer(), abort_flag);
            break;
          }
        }
        const int acc = turn & 1;
        const uint32_t idesc = ptx::idesc_nvfp4(mma_columns(valid_columns(u, TILE)));
        if (!ptx::mbar_wait_bounded(acc_empty_bar + acc, (uint32_t(turn >> 1) & 1u) ^ 1u)) {
          report(p.error, 0x28000000u | (blockIdx.x << 8) | acc, abort_flag);
          break;
        }
        if (!ptx::mbar_wait_bounded(sf_ready_bar + slot.at, slot.phase)) {
          report(p.error, 0x37000000u | (blockIdx.x << 8) | slot.at, abort_flag);
          break;
        }
        const uint32_t t16 = tok_base16 + uint32_t(rows.buffer()) * uint32_t(C::kTokBytes >> 4);
        const uint32_t sfw = tmem_base + C::kSfWgtCol + uint32_t(slot.at) * C::kSfSlotCols;
        const uint32_t sft = tmem_base + C::kSfTokCol + uint32_t(rows.buffer()) * C::kSfSlotCols;
#pragma unroll
        for (int j = 0; j < C::kSlabs; ++j) {
          if (!ptx::mbar_wait_bounded(full_bar + slab.at, slab.phase)) {
            report(p.error, 0x38000000u | (blockIdx.x << 8) | slab.at, abort_flag);
            failed = true;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t w16 = smem_base16 + uint32_t(slab.at) * uint32_t(C::kWgtSlab >> 4);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int kb = 4 * j + i;
            if (kb < C::kKBlocks)
              ptx::tc_mma_nvfp4(tmem_base + acc * TILE, make_desc(w16 + 2 * i), make_desc(t16 + uint32_t(j) * (C::kTokSlab >> 4) + 2 * i),
                                idesc, sfw + 4 * kb, sft + 4 * kb, kb != 0 ? 1u : 0u);
          }
          ptx::tc_commit(empty_bar + slab.at);
          slab.step(C::kRing);
        }
        if (failed) break;
        ptx::tc_commit(sf_empty_bar + slot.at);
        ptx::tc_commit(acc_full_bar + acc);
        slot.step(C::kSfSlots);
      }
    }
    __syncwarp();
  } else if (warp < kFirstEpilogueWarp) {
    // ------------------------------------------------------------------ scale loaders
    const uint32_t quad_lane = uint32_t((warp % 4) * 32) << 16;
    // 12 atoms of 512 bytes (the twelfth is never read by an MMA) -> 48 tensor-memory columns
    auto copy_scales = [&](const uint8_t* atoms, uint32_t column, uint32_t sub) {
      const uint32_t src = ptx::smem_u32(atoms) + lane * 16;
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        uint32_t r[16];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const uint4 v = rotated(ptx::lds128(src + (4 * g + a) * 512), sub);
          r[4 * a] = v.x; r[4 * a + 1] = v.y; r[4 * a + 2] = v.z; r[4 * a + 3] = v.w;
        }
        ptx::tmem_store16(tmem_base + column + 16 * g + quad_lane, r);
      }
      ptx::tmem_store_wait();
      ptx::tc_fence_before_sync();
      __syncwarp();
    };
    Cursor slot;
    Rows rows;
    Unit u{-1, 0, 0, 0, 0};
    for (int w = range.begin; w < range.end && !*abort_flag; ++w) {
      decode_unit(table, w, C::kCTiles, u);
      if (rows.changed(u)) {
        const int buffer = rows.buffer();
        // one barrier covers the rows and their scale atoms
        if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(tok_full_bar + buffer, rows.phase()))) {
          report(p.error, 0x6a000000u | (blockIdx.x << 8) | buffer, abort_flag);
          break;
        }
        copy_scales(token_buf + buffer * C::kTokBytes + C::kSlabs * C::kTokSlab, C::kSfTokCol + uint32_t(buffer) * C::kSfSlotCols,
                    TILE < 128 ? uint32_t(u.tile * TILE % 128) / 32 : 0);
        if (lane == 0) ptx::mbar_arrive(tok_ready_bar + buffer);
      }
      if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(sf_full_bar + slot.at, slot.phase))) {
        report(p.error, 0x6b000000u | (blockIdx.x << 8) | slot.at, abort_flag);
        break;
      }
      copy_scales(sf_buf + slot.at * C::kSfRoom, C::kSfWgtCol + uint32_t(slot.at) * C::kSfSlotCols, 0);
      if (lane == 0) ptx::mbar_arrive(sf_ready_bar + slot.at);
      slot.step(C::kSfSlots);
    }
  } else {
    // ------------------------------------------------------------------ epilogue (128 channels x the tile's tokens)
    const int quad = warp % 4, which = (warp - kFirstEpilogueWarp) / 4;      // lanes; every second or fourth chunk of 16 tokens
    Unit u{-1, 0, 0, 0, 0};
    float alpha = 0.0F;
    int info_of = -1, turn = 0;
    bf16* out = static_cast<bf16*>(p.out);
    for (int w = range.begin; w < range.end && !*abort_flag; ++w, ++turn) {
      decode_unit(table, w, C::kCTiles, u);
      if (info_of != u.e) {
        alpha = p.experts[u.e].alpha[2];
        info_of = u.e;
      }
      const int acc = turn & 1;
      const int valid = valid_columns(u, TILE);
      const size_t row0 = size_t(u.first) + u.tile * TILE;
      const int channel = u.part * 128 + quad * 32 + lane;
      if (!ptx::mbar_wait_warp(acc_full_bar + acc, uint32_t(turn >> 1) & 1u)) {
        report(p.error, 0x47000000u | (blockIdx.x << 8) | acc, abort_flag);
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + acc * TILE + (uint32_t(quad * 32) << 16);
      // A lane has one channel of sixteen tokens.  It stores them one by one, the warp 64 contiguous bytes of a token: as many
      // passes through the L1 data pipe as 16-byte stores of transposed values, without the shuffles.  (16-byte stores whose
      // neighbouring lanes lie in different rows took twice as many: 1500 rows, skewed, down 76 -> 68 us.)
#pragma unroll 1
      for (int c0 = which * 16; c0 < valid; c0 += kEpilogueWarps<TILE> * 4) {
        uint32_t r[16];
        ptx::tmem_load16(taddr + c0, r);
        ptx::tmem_load_wait();
        bf16* dst = out + (row0 + c0) * size_t(kHidden) + channel;
        if (p.row_dest == nullptr) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (c0 + i < valid) dst[i * kHidden] = __float2bfloat16_rn(__fmul_rn(__uint_as_float(r[i]), alpha));
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (c0 + i < valid) {
              bf16* home = reinterpret_cast<bf16*>(p.row_dest[row0 + c0 + i]);         // the row's home, perhaps another GPU
              if (home != nullptr) home[channel] = __float2bfloat16_rn(__fmul_rn(__uint_as_float(r[i]), alpha));
            }
        }
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(acc_empty_bar + acc);
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <typename Kernel>
cudaError_t launch_instance(Kernel kernel, int threads, int smem_bytes, bool* configured_on, const PairMoeParams& params, int sm_count, cudaStream_t stream) {
  bool& configured = configured_on[current_device_slot()];      // the attribute is per GPU (and per instantiation)
  if (!configured) {
    const cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
    if (status != cudaSuccess) return status;
    configured = true;
  }
  return launch_pdl_shared(kernel, dim3(sm_count), dim3(threads), size_t(smem_bytes), stream, params);
}

}  // namespace

cudaError_t launch_moe_narrow_gate_up(int tile_rows, const PairMoeParams& params, int sm_count, cudaStream_t stream) {
  static bool configured[2][kMaxDeviceSlots] = {};
  switch (tile_rows) {
    case 64: return launch_instance(moe_narrow_gate_up_kernel<64>, kThreads<64>, GateUp<64>::kSmemBytes, configured[0], params, sm_count, stream);
    case 128: return launch_instance(moe_narrow_gate_up_kernel<128>, kThreads<128>, GateUp<128>::kSmemBytes, configured[1], params, sm_count, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_moe_narrow_down(int tile_rows, const PairMoeParams& params, int sm_count, cudaStream_t stream) {
  static bool configured[2][kMaxDeviceSlots] = {};
  switch (tile_rows) {
    case 64: return launch_instance(moe_narrow_down_kernel<64>, kThreads<64>, Down<64>::kSmemBytes, configured[0], params, sm_count, stream);
    case 128: return launch_instance(moe_narrow_down_kernel<128>, kThreads<128>, Down<128>::kSmemBytes, configured[1], params, sm_count, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace gw
