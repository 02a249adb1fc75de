// FP8 and BF16 prefill GEMM on CTA pairs (tcgen05 cta_group::2, kind::f8f6f4 / kind::f16) for sm_100a.
//
// What bounds it: the tensor pipe, if it can be fed.  A single CTA with a 128 x 256 tile brings 48 KB through
// L2 -> shared memory for 512 cycles of MMA; two CTAs that share the token tile (each stages its own 128 weight rows
// and half of the tokens, the pair's tensor cores read both halves) need 32 KB each.  Without block scales tensor
// memory has room for two 256-column accumulators, so a tile's epilogue runs under the next tile's MMAs.  Channels
// are on the lanes because their number is a multiple of 128 while the tokens are not: the column width of a tile
// goes in steps of 32, so that 1025 tokens cost 1120 (5 x 224) and not 1280.
// Measured (us, with the activation quantiser): FP8 2048x5376x43008 653 -> 341 (with half of the loads left out 301),
// 1025x5376x16384 113 -> 81; BF16 4096x2816x4096 84 -> 68, 200x2816x8192 26.2 -> 15.3.
//
// Roles per CTA: warp 0 = producer (one lane), warp 1 = MMA issuer (one lane, only in the pair's leader), warps
// 4..11 = epilogue.
// The GeGLU form computes gate and up of 64 channels per CTA and writes their GeGLU, as E4M3 where an FP8 projection takes it:
// BF16 [rows, gate | up] is neither written nor read.  MLP, us, before / after: FP8 5376 -> 21504 276 rows 139 / 134, 2048 673 /
// 607, 2560 -> 7040 1923 rows 123 / 105; BF16 5376 -> 21504 1024 rows 626 / 591.
// Cross-CTA protocol (barriers at the same offsets in both CTAs):
//   full[s]   in the leader; the operand tiles of both CTAs complete on it (the peer's copies into the peer's own
//             shared memory may count there before the leader expects them: only its arrival closes the phase)
//   empty[s], acc_full[a]   local; signalled in both CTAs at once by the leader's tcgen05.commit
//   acc_empty[a]   in the leader, 16 arrivals (epilogue warps of both CTAs)
// The split form is for a few tiles with a long K: two to four pairs in one cluster each have a part of a tile's K slabs and add
// their FP32 sums up through each other's shared memory (BF16 401x6480x560 22.6 -> 12.1 us).
// Every wait is bounded; the kernel ends with a cluster barrier before tensor memory is released.  No load fans
// out to other CTAs.
#include "common.cuh"
#include "gemm_pair_wide.h"
#include "pair.cuh"
#include "ptx.cuh"

namespace gw {
namespace {

using namespace pair;

constexpr int kMaxStages = 12;
constexpr int kWgtBytes = 128 * 128;
constexpr int kEpilogueWarps = 8, kFirstEpilogueWarp = 4;
constexpr int kThreads = 32 * (kFirstEpilogueWarp + kEpilogueWarps);
constexpr int kAccCols = 256, kTmemCols = 512;
// The GeGLU form's epilogue transposes through shared memory: each half of its warps 32 tokens of [gate 64 | up 64] BF16 values,
// 16 bytes more against bank conflicts.
constexpr int kPitch = 256 + 16, kStagingBytes = 32 * kPitch;
constexpr int ring_bytes(bool geglu) { return 221 * 1024 - (geglu ? 2 * kStagingBytes : 0); }
constexpr int kSmemBytes = 221 * 1024 + 1024;
constexpr int kPartCols = 128;                     // the GeGLU form's accumulators of a part of K
static_assert(4 * kPartCols <= kTmemCols, "tensor memory over-subscribed");
constexpr int kMaxSplit = 4;
constexpr int kPartBytes = 128 * 32 * 4;             // one pair's FP32 part of 32 tokens
static_assert(4 * kPartBytes <= ring_bytes(false) && 3 * 2 * kPartBytes <= ring_bytes(false) && 2 * 3 * kPartBytes <= ring_bytes(false),
              "the parts that a pair sums in a split by two, three and four");
enum class WideOut { store, split, geglu, geglu_fp8 };
constexpr int kGroupTiles = 8;                     // token tiles that are walked together
constexpr uint32_t kDescHiSw128 = uint32_t(1024 >> 4) | (1u << 14) | (2u << 29);   // SBO 1024 B, version 1, SWIZZLE_128B

__device__ __forceinline__ uint64_t make_desc(uint32_t lo16) { return (uint64_t(kDescHiSw128) << 32) | lo16; }

// copy into this CTA's shared memory that completes on a barrier of the pair's leader
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* map, int32_t x, int32_t y, uint32_t leader_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(ptx::smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(leader_bar) : "memory");
}

template <bool FP8>
__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  if constexpr (FP8)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

// Work item -> tile.  Eight token tiles at a time go through all channels, token tile fastest: the pairs that run
// together (74) then read 8 token tiles and about 9 weight tiles, whatever the larger side of the problem is.
// The tiles behind the last whole wave are divided into pieces of fewer tokens, so that all pairs have one.
struct Tile { int channel, token0, width, end; };      // first token, token columns, end of the tokens that it stores
__device__ __forceinline__ Tile tile_of(const PairWideTiles& t, int rows, int w) {
  int index = w, piece = 0;
  const bool whole = w < t.whole;
  if (!whole) {
    const int behind = w - t.whole;
    index = t.whole + behind / t.pieces;
    piece = behind % t.pieces;
  }
  const int group = index / (kGroupTiles * t.channel_tiles);
  const int rest = index - group * kGroupTiles * t.channel_tiles;
  const int across = min(kGroupTiles, t.token_tiles - group * kGroupTiles);
  const int tile0 = (group * kGroupTiles + rest % across) * t.tile_rows;
  const int width = whole ? t.tile_rows : t.piece_rows;
  const int token0 = tile0 + piece * width;
  return {rest / across, token0, width, min(min(token0 + width, tile0 + t.tile_rows), rows)};
}
__host__ __device__ __forceinline__ int work_items(const PairWideTiles& t) {
  return t.whole + (t.channel_tiles * t.token_tiles - t.whole) * t.pieces;
}

// barrier of one half of the epilogue warps with a vote: whether one of its threads gave up, so that all of them leave together
__device__ __forceinline__ bool half_barrier_any(int half, bool failed) {
  uint32_t any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(any) : "r"(uint32_t(failed)), "r"(1 + half) : "memory");
  return any != 0;
}
__device__ __forceinline__ void half_barrier(int half) { asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory"); }

template <bool FP8, WideOut OUT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_pair_wide_kernel(const __grid_constant__ PairWideParams p) {
  constexpr bool kGeglu = OUT == WideOut::geglu || OUT == WideOut::geglu_fp8, kSplit = OUT == WideOut::split;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], acc_full_bar[2], acc_empty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x) / 32, 0), lane = threadIdx.x % 32;
  // Rank in the pair (0 = leader) and the leader's in the cluster; a cluster is one pair, or p.tiles.split of them.
  const uint32_t cta = cluster_rank(), rank = kSplit ? cta & 1u : cta, leader = kSplit ? cta & ~1u : 0u;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxStages; ++s) {
      ptx::mbar_init(full_bar + s, 1);
      ptx::mbar_init(empty_bar + s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(acc_full_bar + a, 1);
      ptx::mbar_init(acc_empty_bar + a, 2 * kEpilogueWarps);
    }
    abort_flag = 0;
    ptx::fence_barrier_init();
    ptx::fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_slot, kTmemCols);
    tmem_relinquish_pair();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                               // both CTAs' barriers exist before anybody signals them
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_slot, 0);
  griddep_enter();
  const int pairs = kSplit ? gridDim.x / (2 * p.tiles.split) : gridDim.x / 2, pair = kSplit ? blockIdx.x / (2 * p.tiles.split) : blockIdx.x / 2;
  const int total_work = work_items(p.tiles);
  // Split: one tile per cluster, an even part of its K slabs per pair
  const int first_ks = kSplit ? int(leader / 2) * p.k_stages / p.tiles.split : 0;
  const int end_ks = kSplit ? int(leader / 2 + 1) * p.k_stages / p.tiles.split : p.k_stages;
  // GeGLU of at most one tile a pair, 128 tokens wide at most: tensor memory holds four accumulators, each for an even part of K,
  // and the epilogue adds them up.  The swap form, which runs such rows otherwise, divides K over four CTAs, and a sum of all of K
  // in one accumulator is further from the exact one (outputs that are not the nearest BF16, 2816 -> 2176, swap form / one
  // accumulator: BF16 16 rows 4.1e-4 / 1.5e-3, FP8 with blocks of sixteen activations scaled by 2^-6 .. 2^6 1.7e-4 / 5.5e-4).
  const bool quarters = kGeglu && total_work <= pairs && p.tiles.tile_rows <= kPartCols && p.k_stages >= 4;

  if (warp == 0) {
    // ------------------------------------------------------------------ producer (one lane)
    if (ptx::elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      const uint32_t leader_full = cluster_address(full_bar, leader);
      for (int w = pair; w < total_work && !abort_flag; w += pairs) {
        const Tile tile = tile_of(p.tiles, p.rows, w);
        // GeGLU: 64 gate rows, then the up rows of the same channels
        const int weight_row = (tile.channel * 2 + int(rank)) * (kGeglu ? 64 : 128);
        const int token_row = tile.token0 + int(rank) * (tile.width / 2);
        const uint32_t bytes = 2 * (kWgtBytes + uint32_t(tile.width / 2) * 128);  // of both CTAs
        const CUtensorMap* map_tokens = w < p.tiles.whole ? &p.map_tokens : &p.map_piece;
        bool failed = false;
        for (int ks = first_ks; ks < end_ks; ++ks) {
          if (!ptx::mbar_wait_bounded(empty_bar + stage, phase ^ 1)) {
            report(p.error, 0x15000000u | (blockIdx.x << 8) | stage, &abort_flag);
            failed = true;
            break;
          }
          uint8_t* base = smem + stage * p.stage_bytes;
          if (rank == 0) ptx::mbar_expect_tx(full_bar + stage, bytes);       // rows beyond a matrix arrive as zeros
          tma_load_pair(base, &p.map_weights, ks * 128, weight_row, leader_full + stage * 8);
          if constexpr (kGeglu) tma_load_pair(base + kWgtBytes / 2, &p.map_up, ks * 128, weight_row, leader_full + stage * 8);
          tma_load_pair(base + kWgtBytes, map_tokens, ks * 128, token_row, leader_full + stage * 8);
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
        if (failed) break;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA, whole warp)
    if (rank == 0) {
      int stage = 0, turn = 0;
      uint32_t phase = 0;
      // FP32 accumulator, E4M3 or BF16 operands, M = 256 across the pair
      const uint32_t idesc_of_width = (1u << 4) | (FP8 ? 0u : (1u << 7) | (1u << 10)) | ((256u >> 4) << 24);
      const uint32_t smem_base16 = ptx::smem_u32(smem) >> 4;
      bool failed = false;
      for (int w = pair; w < total_work && !failed; w += pairs, ++turn) {
        const int acc = turn & 1;
        if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(acc_empty_bar + acc, (uint32_t(turn >> 1) & 1u) ^ 1u))) {
          report(p.error, 0x25000000u | (blockIdx.x << 8) | acc, &abort_flag);
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t d = tmem_base + acc * kAccCols;
        const uint32_t idesc = idesc_of_width | ((uint32_t(w < p.tiles.whole ? p.tiles.tile_rows : p.tiles.piece_rows) >> 3) << 17);
        // The split form has both accumulators to itself: each takes half of the K slabs.
        const int mid_ks = kSplit ? (first_ks + end_ks + 1) / 2 : end_ks;
        int part = 0, part_end = quarters ? p.k_stages / 4 : p.k_stages;
        bool begins = true;
        for (int ks = first_ks; ks < end_ks; ++ks) {
          if (kGeglu && ks == part_end) {
            begins = true;
            part_end = (++part + 1) * p.k_stages / 4;
          }
          if (!__all_sync(0xffffffffu, ptx::mbar_wait_bounded(full_bar + stage, phase))) {
            report(p.error, 0x35000000u | (blockIdx.x << 8) | stage, &abort_flag);
            failed = true;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t base16 = smem_base16 + uint32_t(stage) * (uint32_t(p.stage_bytes) >> 4);
          if (ptx::elect_one()) {
            const int nkb = ks + 1 == p.k_stages ? p.last_kb : 4;
            const uint64_t a = make_desc(base16), b = make_desc(base16 + (kWgtBytes >> 4));
#pragma unroll
            for (int kb = 0; kb < 4; ++kb)
              if (kb < nkb) {
                if constexpr (kGeglu)
                  mma_pair<FP8>(d + uint32_t(part * kPartCols), a + 2 * kb, b + 2 * kb, idesc, begins && kb == 0 ? 0u : 1u);
                else
                  mma_pair<FP8>(kSplit && ks >= mid_ks ? d + kAccCols : d, a + 2 * kb, b + 2 * kb, idesc,
                                ((kSplit && ks >= mid_ks ? ks - mid_ks : ks - first_ks) | kb) != 0 ? 1u : 0u);
              }
            commit_pair(empty_bar + stage, leader);
          }
          __syncwarp();
          begins = false;
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
        if (!failed && ptx::elect_one()) commit_pair(acc_full_bar + acc, leader);
      }
    }
    __syncwarp();
  } else if (kGeglu && warp >= kFirstEpilogueWarp) {
    // ------------------------------------------------------------------ epilogue: GeGLU (own 64 channels x tile_rows tokens)
    // The gate lanes (0..63) and the up lanes (64..127) of a channel belong to different warps: the scaled accumulators, rounded
    // to BF16, which is what GeGLU consumes, go through shared memory; then a thread has sixteen channels of a token.
    const int quad = warp % 4;
    const int half = (warp - kFirstEpilogueWarp) / 4;            // takes every other 32-token chunk
    const uint32_t leader_acc_empty = leader_address(acc_empty_bar);
    uint8_t* staging = smem + ring_bytes(true) + half * kStagingBytes;
    const int tid = (int(threadIdx.x) - 32 * kFirstEpilogueWarp) % 128;
    const float* channel_alpha = quad < 2 ? p.channel_alpha : p.channel_alpha_up;
    int turn = 0;
    for (int w = pair; w < total_work; w += pairs, ++turn) {
      const int acc = turn & 1;
      const Tile tile = tile_of(p.tiles, p.rows, w);
      const int channel0 = (tile.channel * 2 + int(rank)) * 64;
      const int mine = channel0 + quad % 2 * 32 + lane;
      const float scale = channel_alpha == nullptr ? (quad < 2 ? p.alpha : p.alpha_up) : mine < p.n ? __ldg(channel_alpha + mine) : 0.0F;
      const bool arrived = ptx::mbar_wait_warp(acc_full_bar + acc, uint32_t(turn >> 1) & 1u);
      if (!arrived) report(p.error, 0x4b000000u | (blockIdx.x << 8) | acc, &abort_flag);
      if (half_barrier_any(half, !arrived)) break;
      ptx::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + acc * kAccCols + (uint32_t(quad * 32) << 16);
      for (int t0 = half * 32; t0 < tile.width; t0 += 64) {
        const int token0 = tile.token0 + t0;
        if (token0 >= tile.end) break;                                // the whole half
        uint32_t r[32];
        if (quarters) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t q[4][16];
#pragma unroll
            for (int part = 0; part < 4; ++part) ptx::tmem_load16(taddr + part * kPartCols + t0 + 16 * h, q[part]);
            ptx::tmem_load_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i)
              r[16 * h + i] = __float_as_uint(__uint_as_float(q[0][i]) + __uint_as_float(q[1][i]) + __uint_as_float(q[2][i]) + __uint_as_float(q[3][i]));
          }
        } else {
          ptx::tmem_load16(taddr + t0, r);
          ptx::tmem_load16(taddr + t0 + 16, r + 16);
          ptx::tmem_load_wait();
        }
        if (t0 != half * 32) half_barrier(half);                    // the chunk before has been read
        uint16_t* put = reinterpret_cast<uint16_t*>(staging) + quad * 32 + lane;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const bf16 v = __float2bfloat16_rn(__fmul_rn(__uint_as_float(r[i]), scale));
          put[i * (kPitch / 2)] = *reinterpret_cast<const uint16_t*>(&v);
        }
        half_barrier(half);
        const int token = token0 + tid / 4, channel = channel0 + tid % 4 * 16;
        if (token >= tile.end || channel >= p.n) continue;
        const uint32_t from = ptx::smem_u32(staging) + uint32_t(tid / 4) * kPitch + uint32_t(tid % 4) * 32;
        uint32_t words[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 g = ptx::lds128(from + 16 * h), u = ptx::lds128(from + 128 + 16 * h);
          const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float lo = gelu_tanh_multiply_bf16(__uint_as_float(gw[i] << 16), __uint_as_float(uw[i] << 16));
            const float hi = gelu_tanh_multiply_bf16(__uint_as_float(gw[i] & 0xFFFF0000u), __uint_as_float(uw[i] & 0xFFFF0000u));
            if constexpr (OUT == WideOut::geglu_fp8)
              words[4 * h + i] = __nv_cvt_float2_to_fp8x2(make_float2(__fmul_rn(lo, p.inverse_scale), __fmul_rn(hi, p.inverse_scale)), __NV_SATFINITE, __NV_E4M3);
            else
              words[4 * h + i] = (__float_as_uint(lo) >> 16) | (__float_as_uint(hi) & 0xFFFF0000u);
          }
        }
        if constexpr (OUT == WideOut::geglu_fp8) {
          *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.out) + size_t(token) * p.ld_out + channel) =
              make_uint4(words[0] | words[1] << 16, words[2] | words[3] << 16, words[4] | words[5] << 16, words[6] | words[7] << 16);
        } else {
          uint4* dst = reinterpret_cast<uint4*>(static_cast<bf16*>(p.out) + size_t(token) * p.ld_out + channel);
          dst[0] = make_uint4(words[0], words[1], words[2], words[3]);
          dst[1] = make_uint4(words[4], words[5], words[6], words[7]);
        }
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive_cluster(leader_acc_empty + acc * 8);
    }
  } else if (kSplit && warp >= kFirstEpilogueWarp) {
    if (!ptx::mbar_wait_warp(acc_full_bar, 0)) report(p.error, 0x55000000u | (blockIdx.x << 8), &abort_flag);
  } else if (warp >= kFirstEpilogueWarp) {
    // ------------------------------------------------------------------ epilogue (own 128 channels x tile_rows tokens)
    const int quad = warp % 4;
    const int half = (warp - kFirstEpilogueWarp) / 4;            // takes every other 32-token chunk
    const uint32_t leader_acc_empty = leader_address(acc_empty_bar);
    bf16* out = static_cast<bf16*>(p.out);
    int turn = 0;
    for (int w = pair; w < total_work && !abort_flag; w += pairs, ++turn) {
      const int acc = turn & 1;
      const Tile tile = tile_of(p.tiles, p.rows, w);
      const int channel0 = (tile.channel * 2 + int(rank)) * 128 + quad * 32;
      const float scale = p.channel_alpha == nullptr ? p.alpha : channel0 + lane < p.n ? __ldg(p.channel_alpha + channel0 + lane) : 0.0F;
      if (!ptx::mbar_wait_warp(acc_full_bar + acc, uint32_t(turn >> 1) & 1u)) {
        report(p.error, 0x45000000u | (blockIdx.x << 8) | acc, &abort_flag);
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + acc * kAccCols + (uint32_t(quad * 32) << 16);
      // A lane has one channel of 32 tokens and stores them one by one, the warp 64 contiguous bytes of a token.
      const bool inside = channel0 + lane < p.n;
      for (int t0 = half * 32; t0 < tile.width; t0 += 64) {
        const int token0 = tile.token0 + t0;
        if (token0 >= tile.end) break;                                // warp-uniform
        uint32_t r[32];
        ptx::tmem_load16(taddr + t0, r);
        ptx::tmem_load16(taddr + t0 + 16, r + 16);
        ptx::tmem_load_wait();
        bf16* dst = out + size_t(token0) * p.ld_out + channel0 + lane;
        const int left = inside ? tile.end - token0 : 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (i < left) *dst = __float2bfloat16_rn(__fmul_rn(__uint_as_float(r[i]), scale));
          dst += p.ld_out;
        }
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive_cluster(leader_acc_empty + acc * 8);
    }
  }

  if constexpr (kSplit) {
    // ------------------------------------------------------------------ sum of the pairs' parts
    // Chunk c of 32 tokens is summed and stored by pair c % split: the other pairs write their 128 x 32 FP32 values of it into
    // that pair's operand ring, [token / 4][lane][token % 4], once every pair's MMAs have read theirs.
    __syncwarp();
    const int split = p.tiles.split;
    if (split > 1) {
      ptx::tc_fence_before_sync();
      cluster_sync_all();
    }
    ptx::tc_fence_after_sync();
    const int part = int(leader / 2), quad = warp % 4, half = (warp - kFirstEpilogueWarp) / 4;
    const Tile tile = tile_of(p.tiles, p.rows, pair);
    const int chunks = (tile.end - tile.token0 + 31) / 32;
    const uint32_t taddr = tmem_base + (uint32_t(quad * 32) << 16);
    const uint32_t at = uint32_t(quad * 32 + lane) * 16;
    const bool both = end_ks - first_ks > 1;           // accumulators
    const auto load_sum = [&](int c, uint32_t* r) {
      ptx::tmem_load16(taddr + 32 * c, r);
      ptx::tmem_load16(taddr + 32 * c + 16, r + 16);
      if (both) {
        uint32_t s[32];
        ptx::tmem_load16(taddr + kAccCols + 32 * c, s);
        ptx::tmem_load16(taddr + kAccCols + 32 * c + 16, s + 16);
        ptx::tmem_load_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + __uint_as_float(s[i]));
      } else {
        ptx::tmem_load_wait();
      }
    };
    if (split > 1 && warp >= kFirstEpilogueWarp) {
      for (int c = half; c < chunks; c += 2) {
        const int owner = c % split;
        if (owner == part) continue;
        uint32_t r[32];
        load_sum(c, r);
        const int slot = c / split * (split - 1) + (part < owner ? part : part - 1);
        const uint32_t to = cluster_address(smem + slot * kPartBytes, uint32_t(2 * owner) + rank) + at;
#pragma unroll
        for (int i = 0; i < 8; ++i) store_cluster(to + i * (128 * 16), r + 4 * i);
      }
    }
    __syncwarp();
    if (split > 1) cluster_sync_all();
    if (warp >= kFirstEpilogueWarp && !abort_flag) {
      const int channel = (tile.channel * 2 + int(rank)) * 128 + quad * 32 + lane;
      const float scale = p.channel_alpha == nullptr ? p.alpha : channel < p.n ? __ldg(p.channel_alpha + channel) : 0.0F;
      for (int k = half, c = part + half * split; c < chunks; k += 2, c += 2 * split) {
        uint32_t r[32];
        load_sum(c, r);
        for (int other = 0; other < split - 1; ++other) {
          const uint32_t from = ptx::smem_u32(smem + (k * (split - 1) + other) * kPartBytes) + at;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 v = ptx::lds128(from + i * (128 * 16));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) r[4 * i + j] = __float_as_uint(__uint_as_float(r[4 * i + j]) + __uint_as_float(w[j]));
          }
        }
        bf16* dst = static_cast<bf16*>(p.out) + size_t(tile.token0 + 32 * c) * p.ld_out + channel;
        const int left = channel < p.n ? tile.end - tile.token0 - 32 * c : 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          if (i < left) *dst = __float2bfloat16_rn(__fmul_rn(__uint_as_float(r[i]), scale));
          dst += p.ld_out;
        }
      }
    }
    __syncwarp();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                               // the peer no longer reads this CTA's shared or tensor memory
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

template <bool FP8, WideOut OUT>
cudaError_t launch_instance(const PairWideParams& params, int sm_count, cudaStream_t stream) {
  static bool configured_on[kMaxDeviceSlots] = {};   // the attribute is per GPU
  bool& configured = configured_on[current_device_slot()];
  if (!configured) {
    const cudaError_t status = cudaFuncSetAttribute(gemm_pair_wide_kernel<FP8, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (status != cudaSuccess) return status;
    configured = true;
  }
  const int work = work_items(params.tiles), split = params.tiles.split;
  const int pairs = split > 0 ? work * split : work < sm_count / 2 ? work : sm_count / 2;
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(2 * pairs);
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = kSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attributes[2]{};
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = split > 0 ? 2 * split : 2;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = 2;
  note_launch();
  return cudaLaunchKernelEx(&config, gemm_pair_wide_kernel<FP8, OUT>, params);
}

}  // namespace

PairWideTiles pair_wide_tiles(uint32_t rows, uint32_t n, int k_stages, int sm_count) {
  // A tile takes as long as its weight rows and MMA issue cost whatever its width (about 136 columns) plus its columns:
  // measured on FP8 K=5376, per wave of tiles of 64 / 128 / 192 / 256 tokens 8.9 / 11.3 / 14.3 / 17.4 us.
  const int channel_tiles = int((n + 255) / 256), pairs = sm_count / 2;
  const bool small = rows <= 128 && k_stages > 0;
  PairWideTiles t{};
  uint64_t best_cost = ~0ull;
  for (int tile = small ? 128 : 256; tile >= (small ? 32 : 64); tile -= 32) {
    const int token_tiles = int((rows + tile - 1) / tile);
    const uint64_t tiles = uint64_t(channel_tiles) * token_tiles;
    const uint64_t cost = (tiles + pairs - 1) / pairs * uint64_t(tile + 136);
    if (cost < best_cost && (!small || tiles <= uint64_t(pairs))) {
      best_cost = cost;
      t = {tile, channel_tiles, token_tiles, int32_t(tiles), 1, tile, small ? 1 : 0};
    }
  }
  // K shared by the pairs of a cluster, where few wide tiles leave pairs idle and narrower ones would read the weights more often: a
  // slab of a tile costs what it did, the launch and its barriers about 900 columns more, and 20 per column whose sum another pair
  // has.  It has to win an eighth, because pairs at work slow each other down.  us, one pair / several, quantiser included: FP8
  // 218x16384x5376 (three pairs, 224 wide) 32.9 / 27.4, 130x21504x5376 38.9 / 29.1, 180x8192x2816 18.0 / 13.4, BF16 140x5376x2048
  // 19.7 / 12.2, 250x5376x4096 (two, 128 wide) 20.8 / 16.4; outside of the rule BF16 200x2816x8192 14.4 / 16.7, 491x5376x4096
  // 22.2 / 23.0, FP8 300x2816x2816 9.6 / 10.1, 800x5376x2048 16.0 / 17.2.
  uint64_t split_cost = (best_cost * uint64_t(k_stages) + 1900) * 7 / 8;
  for (int split = 2; split <= kMaxSplit && split <= k_stages; ++split)
    for (int tile = small ? 128 : 256; tile >= (small ? 32 : 64); tile -= 32) {
      const int token_tiles = int((rows + tile - 1) / tile);
      const uint64_t tiles = uint64_t(channel_tiles) * token_tiles;
      const uint64_t cost = uint64_t((k_stages + split - 1) / split) * uint64_t(tile + 136) + 2800 + uint64_t(20 * tile * (split - 1) / split);
      if (cost < split_cost && tiles * split <= uint64_t(pairs) && int64_t(tiles) <= clusters_at_once<gemm_pair_wide_kernel<true, WideOut::split>>(split, kThreads, kSmemBytes)) {
        split_cost = cost;
        t = {tile, channel_tiles, token_tiles, int32_t(tiles), 1, tile, split};
      }
    }
  if (t.split > 0) return t;
  // A last wave for half of the pairs or fewer: its tiles in as many pieces as keep every pair at work, 32 columns or a multiple.
  // us, whole tiles / pieces: FP8 250x5376x21504 (74 + 10 tiles) 37.2 / 32.9, 180 rows 32.5 / 30.7, BF16 200 rows 59.2 / 55.0,
  // 4096x2816x4096 (222 + 34) 65.1 / 62.5, FP8 1025x5376x16384 (296 + 24) 76.0 / 75.5.  A wave with few tiles is quicker than a
  // full one, so that a tile width chosen for its pieces loses (BF16 2048x2816x2816, 256 wide and four pieces against 160 wide
  // 25.4 / 27.4).
  const int behind = t.whole % pairs;
  if (t.whole > pairs && behind > 0 && behind <= pairs / 2) {
    const int most = pairs / behind;
    t.whole -= behind;
    t.piece_rows = ((t.tile_rows + most - 1) / most + 31) / 32 * 32;
    t.pieces = (t.tile_rows + t.piece_rows - 1) / t.piece_rows;
  }
  return t;
}

namespace {
PairWideParams with_ring(const PairWideParams& given, bool geglu) {
  PairWideParams params = given;
  params.stage_bytes = kWgtBytes + given.tiles.tile_rows * 64;
  const int fit = ring_bytes(geglu) / params.stage_bytes;
  params.stages = fit < kMaxStages ? fit : kMaxStages;
  return params;
}
}  // namespace

cudaError_t launch_gemm_pair_wide(bool fp8, const PairWideParams& given, int sm_count, cudaStream_t stream) {
  const PairWideParams params = with_ring(given, false);
  if (params.tiles.split > 0)
    return fp8 ? launch_instance<true, WideOut::split>(params, sm_count, stream) : launch_instance<false, WideOut::split>(params, sm_count, stream);
  return fp8 ? launch_instance<true, WideOut::store>(params, sm_count, stream) : launch_instance<false, WideOut::store>(params, sm_count, stream);
}

cudaError_t launch_gemm_pair_wide_geglu(bool fp8, bool quantise, const PairWideParams& given, int sm_count, cudaStream_t stream) {
  const PairWideParams params = with_ring(given, true);
  if (quantise)
    return fp8 ? launch_instance<true, WideOut::geglu_fp8>(params, sm_count, stream) : launch_instance<false, WideOut::geglu_fp8>(params, sm_count, stream);
  return fp8 ? launch_instance<true, WideOut::geglu>(params, sm_count, stream) : launch_instance<false, WideOut::geglu>(params, sm_count, stream);
}

}  // namespace gw
