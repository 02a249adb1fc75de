// Weight-streaming projections for small row counts (decode): one launch quantises the
// activations, reads every weight once and writes the BF16 result.
//
// What bounds it: the weight bytes from HBM, and at small sizes latency.  The flat sequence of (block of 32 weight rows, 128-byte
// chunk of K) pieces is cut into ranges, one per SM -- whole row blocks where all of K is one slab, equal ranges cut at any piece
// otherwise -- and inside it one per warp, at any piece.  A warp walks its range alone: it has a ring of two pieces of its own that it
// refills itself by tensor copies as soon as it has multiplied one (144 KB per SM on their way for W4A4, 128 for W8A8,
// 108 for W4A16, 96 for BF16), and it stores the row blocks that are wholly its own straight from registers.  Nothing synchronises while weights stream; the
// first pieces are asked for before the kernel waits for its predecessor.  Row blocks that several warps share
// are added through shared memory at the end, those that several SMs share through L2 by the one that
// arrives last at the block's counter -- always in range order, so results do not depend on who comes last.
//
// Measured on cold weights (us, with everything a call does; activation quantiser + tcgen05 kernel in brackets): NVFP4
// 1x2816x2816 5.3 (6.9), FP8 8x2816x2816 6.5 (7.6); W4A16 MLP of eight rows, 5376 -> 21504, 70 against 285 with dequantised
// weights.
//
// Token values live in shared memory in the order the tensor instruction wants them.  When all of K does
// not fit there, K is cut into slabs, the flat sequence walks slab by slab and every row block has one sum
// per slab.
#include <algorithm>
#include <string>

#include "common.cuh"
#include "decode_stream.h"
#include "ptx.cuh"
#include "stream.cuh"

namespace gw {

bool encode_tensor_map_piece(CUtensorMap* map, const void* base, uint64_t row_bytes, uint64_t rows, std::string* error);
bool encode_tensor_map_atoms(CUtensorMap* map, const void* base, uint64_t atoms, std::string* error);

namespace {

using namespace stream;

struct StreamArgs {
  CUtensorMap weights[2], scales[2];
  float alpha[2];
  const float* channel_alpha[2];
  const bf16* input;
  bf16* out;
  size_t ld_out;
  float* partials;
  int32_t* counters;
  uint8_t *packed, *packed_scales;       // w4a4: where the quantised activations are left as well, or nullptr
  uint32_t* error;
  uint32_t reread;                       // a launch after this one reads the same weights
  uint32_t weights_settled;              // the kernel before this one does not write the weights
  float inverse_scale;
  uint32_t rows, k, n, gelu;
  uint32_t blocks, chunks, chunks_per_slab, slabs, max_units;
  uint32_t range, longer, step;          // steps per SM, of `step` pieces each; the first `longer` SMs have one more
  Divisor by_range, by_range1;           // range, range + 1
  Divisor by_slab, by_chunks, by_last_chunks, by_blocks;   // pieces of a whole slab; chunks of a whole and of the last slab; blocks
};

constexpr int kSharedLimit = 226 * 1024;

// Where the piece ranges lie.  Where they cut row blocks (a step is one piece), piece x belongs to thread block cta_of(x).
__device__ __forceinline__ uint32_t range_begin(const StreamArgs& a, uint32_t cta) { return (cta * a.range + min(cta, a.longer)) * a.step; }
__device__ __forceinline__ uint32_t cta_of(const StreamArgs& a, uint32_t x) {
  const uint32_t cut = a.longer * (a.range + 1);
  return x < cut ? a.by_range1.quotient(x) : a.longer + a.by_range.quotient(x - cut);
}

// A "unit" is one row block of one slab: unit = slab * blocks + block.
struct Unit {
  uint32_t slab, block, begin, chunks;     // its first piece, its pieces
};
__device__ __forceinline__ Unit unit_at(const StreamArgs& a, uint32_t unit) {
  Unit u;
  u.slab = a.by_blocks.quotient(unit);
  u.block = unit - u.slab * a.blocks;
  const uint32_t first = u.slab * a.chunks_per_slab;
  u.chunks = min(a.chunks_per_slab, a.chunks - first);
  u.begin = first * a.blocks + u.block * u.chunks;
  return u;
}
__device__ __forceinline__ uint32_t block_of(const StreamArgs& a, uint32_t slab, uint32_t piece_in_slab) {
  return slab + 1 == a.slabs ? a.by_last_chunks.quotient(piece_in_slab) : a.by_chunks.quotient(piece_in_slab);
}
__device__ __forceinline__ uint32_t unit_of(const StreamArgs& a, uint32_t piece) {
  const uint32_t slab = min(a.by_slab.quotient(piece), a.slabs - 1);
  return slab * a.blocks + block_of(a, slab, piece - slab * a.chunks_per_slab * a.blocks);
}

// Row block `block`: rows 8 i .. 8 i + 7 of the four 32-row groups of a 128-row tile (their NVFP4 block scales are 128
// contiguous bytes per atom).  With two matrices, the same rows of both.
struct BlockPlace {
  uint32_t group, row8;      // first 32-row group, i
  __device__ explicit BlockPlace(uint32_t block) : group(block / 4 * 4), row8(block % 4) {}
  __device__ uint32_t channel(uint32_t g, uint32_t slot) const { return (group + slot) * 32 + row8 * 8 + g; }
};

// FP32 sums of a row block, and a lane's share of them: value i of matrix m, token group nt, register r of the two tiles
// is number (m * NT + nt) * 8 + r.
template <int NT, bool PAIR> constexpr int lane_sums() { return NT * 8 * (PAIR ? 2 : 1); }
template <int NT, bool PAIR> constexpr uint32_t unit_values() { return lane_sums<NT, PAIR>() * 32; }

template <int NT, bool PAIR>
struct Sums { float v[lane_sums<NT, PAIR>()]; };

// With two matrices a loop: a launch finds its instructions in no cache when another kernel ran before it and fetches
// them while its own weights fill the memory system.  GeGLU unrolled at every place that stores cost 8 us of a 32 us launch
// between two other kernels.  (A called function costs more: 1.2 us a launch for its stack.)
template <int NT, bool PAIR>
__device__ __forceinline__ void store_unit(const StreamArgs& a, uint32_t block, uint32_t lane, Sums<NT, PAIR>& sum) {
  const BlockPlace place(block);
#pragma unroll (PAIR ? 1 : 16)
  for (int i = 0; i < NT * 8; ++i) {
    const uint32_t channel = place.channel(lane / 4, uint32_t(i) / 2 % 4), token = uint32_t(i) / 8 * 8 + lane % 4 * 2 + (i & 1);
    if (channel < a.n && token < a.rows) {
      bf16 value = __float2bfloat16_rn(__fmul_rn(sum.v[0], a.channel_alpha[0] != nullptr ? a.channel_alpha[0][channel] : a.alpha[0]));
      if constexpr (PAIR) {
        const float up = __fmul_rn(sum.v[NT * 8], a.channel_alpha[1] != nullptr ? a.channel_alpha[1][channel] : a.alpha[1]);
        value = __float2bfloat16_rn(gelu_tanh_multiply_bf16(__bfloat162float(value), __bfloat162float(__float2bfloat16_rn(up))));
      }
      a.out[token * a.ld_out + channel] = value;
    }
#pragma unroll
    for (int j = 0; j + 1 < lane_sums<NT, PAIR>(); ++j) sum.v[j] = sum.v[j + 1];      // the next one comes to the front
  }
}

template <StreamKind KIND, int NT, bool PAIR>
struct Layout {
  // BF16 tokens take four times the room of FP4 ones: fewer warps (and rings) then keep 8192 values of K in one slab
  static constexpr int kWarps = NT == 1 && (KIND == StreamKind::w4a4 || KIND == StreamKind::w8a8) ? 16 : 12;
  static constexpr int kThreads = 32 * kWarps;
  static constexpr uint32_t kSlots = 2;                                                // pieces in a warp's ring
  static constexpr uint32_t kScaleBytes = nvfp4_weights(KIND) ? kPieceScaleBytes : 0;
  static constexpr uint32_t kRingBytes = kWarps * kSlots * (kPieceBytes + kScaleBytes);
  static constexpr uint32_t kSumBytes = kWarps * unit_values<NT, PAIR>() * 4;                // a row block that the warp before began
  static constexpr uint32_t kChunkBytes = NT * token_chunk_bytes<KIND>();
  static constexpr uint32_t kFixedBytes = kRingBytes + kSumBytes + 1024;               // 1024: the ring's alignment
};

// Token values of one slab into shared memory, all threads.
template <StreamKind KIND, int NT, bool PAIR>
__device__ __forceinline__ void stage_tokens(const StreamArgs& a, uint32_t chunk0, uint32_t chunks, bool publish, uint8_t* tokens) {
  using L = Layout<KIND, NT, PAIR>;
  constexpr uint32_t kChunkGroups = chunk_values(KIND) / 16;
  const uint32_t k0 = chunk0 * chunk_values(KIND);
  const uint32_t groups = min(chunks * chunk_values(KIND), a.k - k0) / 16, items = groups * a.rows;
  const bool gelu = (KIND == StreamKind::w4a4 || KIND == StreamKind::w8a8) && a.gelu;
  // Weights fill the memory system while this runs, so a load takes a microsecond or two: a thread asks for all it can.
  constexpr int kBatch = 6;
  uint32_t token = threadIdx.x / groups, group = threadIdx.x % groups;
  for (uint32_t i0 = threadIdx.x; i0 < items; i0 += L::kThreads * kBatch) {
    uint4 raw[kBatch][2];
    uint32_t at = token, where = group;
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      if (i0 + b * L::kThreads >= items) break;
      const uint4* source = reinterpret_cast<const uint4*>(a.input + size_t(at) * (gelu ? 2 : 1) * a.k + k0 + where * 16);
      raw[b][0] = source[0];
      raw[b][1] = source[1];
      for (where += L::kThreads; where >= groups; where -= groups) ++at;
    }
#pragma unroll
    for (int b = 0; b < kBatch; ++b) {
      if (i0 + b * L::kThreads >= items) break;
      const uint32_t k = k0 + group * 16;
      uint32_t pairs[8] = {raw[b][0].x, raw[b][0].y, raw[b][0].z, raw[b][0].w, raw[b][1].x, raw[b][1].y, raw[b][1].z, raw[b][1].w}, codes[2];
      if (gelu) geglu_pairs(a.input + size_t(token) * 2 * a.k + a.k + k, pairs);
      uint8_t* chunk = tokens + group / kChunkGroups * L::kChunkBytes + token / 8 * token_chunk_bytes<KIND>();
      const uint8_t scale = put_tokens<KIND>(chunk, token, group % kChunkGroups, pairs, a.inverse_scale, codes);
      if (KIND == StreamKind::w4a4 && publish) {
        *reinterpret_cast<uint2*>(a.packed + (size_t(token) * a.k + k) / 2) = make_uint2(codes[0], codes[1]);
        a.packed_scales[scale_offset(token, k / 16, a.k)] = scale;
      }
      for (group += L::kThreads; group >= groups; group -= groups) ++token;
    }
  }
}

// A row block's sums of this SM, one warp.  If the SM covers it only in part (or one slab of it), they go to L2, and the
// SM that arrives last at the row block's counter adds everybody's, slab by slab and in range order.
template <int NT, bool PAIR>
__device__ __forceinline__ void finish_unit(const StreamArgs& a, uint32_t unit, uint32_t unit_first, bool whole, uint32_t lane, Sums<NT, PAIR> sum) {
  constexpr uint32_t kValues = unit_values<NT, PAIR>();
  constexpr int kSums = lane_sums<NT, PAIR>();
  const uint32_t block = unit - a.by_blocks.quotient(unit) * a.blocks;
  if (!whole) {
    float* to = a.partials + (size_t(blockIdx.x) * a.max_units + unit - unit_first) * kValues + lane;
#pragma unroll
    for (int i = 0; i < kSums; ++i) __stcg(to + i * 32, sum.v[i]);
    // lane s knows slab s: whose ranges hold the row block's pieces there
    uint32_t cta_first = 0, parts = 0;
    if (lane < a.slabs) {
      const Unit u = unit_at(a, lane * a.blocks + block);
      cta_first = cta_of(a, u.begin);
      parts = cta_of(a, u.begin + u.chunks - 1) - cta_first + 1;
    }
    const uint32_t need = __reduce_add_sync(0xFFFFFFFFu, parts);
    __threadfence();
    __syncwarp();
    uint32_t is_last = 0;
    if (lane == 0) {
      is_last = atomicAdd(a.counters + block, 1) == int32_t(need - 1) ? 1u : 0u;
      if (is_last) a.counters[block] = 0;                      // ready for the next launch
    }
    if (!__shfl_sync(0xFFFFFFFFu, is_last, 0)) return;
    __threadfence();
#pragma unroll
    for (int i = 0; i < kSums; ++i) sum.v[i] = 0.0F;
#pragma unroll 1
    for (uint32_t s = 0; s < a.slabs; ++s) {
      const uint32_t from = __shfl_sync(0xFFFFFFFFu, cta_first, s), n = __shfl_sync(0xFFFFFFFFu, parts, s);
      // a part's place among its SM's: one lane per part
      uint32_t ordinal_of = 0;
      if (lane < n) ordinal_of = s * a.blocks + block - unit_of(a, range_begin(a, from + lane));
#pragma unroll 1
      for (uint32_t j = 0; j < n; ++j) {
        const uint32_t place = __shfl_sync(0xFFFFFFFFu, ordinal_of, j);
        const float* theirs = a.partials + (size_t(from + j) * a.max_units + place) * kValues + lane;
#pragma unroll
        for (int i = 0; i < kSums; ++i) sum.v[i] += __ldcg(theirs + i * 32);
      }
    }
  }
  store_unit<NT, PAIR>(a, block, lane, sum);
}

// PIECE_SUMS: each piece is summed by itself and the sums are added.  The tensor instruction rounds at every step, and the longer
// it adds up the further it ends (StreamPlan::piece_sums says where that matters).
template <StreamKind KIND, int NT, bool PAIR, bool PIECE_SUMS>
__global__ void __launch_bounds__((Layout<KIND, NT, PAIR>::kThreads), 1)
decode_stream_kernel(const __grid_constant__ StreamArgs a) {
  using L = Layout<KIND, NT, PAIR>;
  constexpr uint32_t kValues = unit_values<NT, PAIR>(), kWarps = L::kWarps, kSlots = L::kSlots;
  extern __shared__ uint8_t stream_smem[];
  __shared__ uint64_t full_bar[L::kWarps * L::kSlots];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(stream_smem) + 1023) & ~uintptr_t(1023));
  uint8_t* ring_scales = ring + kWarps * kSlots * kPieceBytes;
  float* sums = reinterpret_cast<float*>(ring + L::kRingBytes);            // [warp][kValues]
  uint8_t* tokens = ring + L::kRingBytes + L::kSumBytes;
  if (threadIdx.x == 0) {
    ptx::prefetch_tensormap(&a.weights[0]);
    if (nvfp4_weights(KIND)) ptx::prefetch_tensormap(&a.scales[0]);
  }
  const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x / 32, 0), lane = threadIdx.x % 32;
  const uint32_t piece_begin = range_begin(a, blockIdx.x), piece_end = range_begin(a, blockIdx.x + 1);
  const uint32_t unit_first = unit_of(a, piece_begin);
  if (lane == 0) {                        // the ring's barriers are this warp's own
    for (uint32_t s = 0; s < kSlots; ++s) ptx::mbar_init(full_bar + warp * kSlots + s, 1);
    ptx::fence_barrier_init();
    ptx::fence_proxy_async_smem();
  }
  __syncwarp();

  const uint64_t policy = a.reread ? ptx::l2_evict_normal() : ptx::l2_evict_first();
  uint32_t slab_unit = unit_first, turn = 0;                // turn: pieces this warp has multiplied
  for (uint32_t slab_begin = piece_begin; slab_begin < piece_end;) {
    // ---- the pieces of one slab, divided among the warps
    const Unit slab = unit_at(a, slab_unit);
    const uint32_t chunk0 = slab.slab * a.chunks_per_slab, base = chunk0 * a.blocks, chunks = slab.chunks;
    const uint32_t slab_end = min(piece_end, base + a.blocks * chunks), count = slab_end - slab_begin;
    const auto warp_begin = [&](uint32_t w) { return slab_begin + (count * w + kWarps - 1) / kWarps; };   // warp 0 has the first
    const uint32_t begin = warp_begin(warp), end = warp_begin(warp + 1);
    uint32_t block = block_of(a, slab.slab, begin - base), chunk = begin - base - block * chunks;
    const uint32_t begin_chunk = chunk;
    uint32_t next = begin, next_block = block, next_chunk = chunk, next_slot = turn % kSlots, next_matrix = 0;      // the piece to ask for next
    auto request = [&](bool into_l2 = false) {
      const uint32_t matrix = PAIR ? next_matrix : 0;
      if (into_l2) {
        if (next < end && ptx::elect_one()) {
          const BlockPlace at(next_block);
          ptx::tma_prefetch_3d(&a.weights[matrix], int32_t((chunk0 + next_chunk) * 128), int32_t(at.row8 * 8), int32_t(at.group), policy);
          if constexpr (nvfp4_weights(KIND))
            ptx::tma_prefetch_2d(&a.scales[matrix], int32_t(at.row8 * 128), int32_t(at.group / 4 * (a.k / 64) + (chunk0 + next_chunk) * 4),
                                 policy);
        }
      } else if (next < end && ptx::elect_one()) {
        const uint32_t place = warp * kSlots + next_slot;
        uint64_t* bar = full_bar + place;
        const BlockPlace at(next_block);
        ptx::mbar_expect_tx(bar, kPieceBytes + L::kScaleBytes);
        ptx::tma_load_3d(ring + place * kPieceBytes, &a.weights[matrix], int32_t((chunk0 + next_chunk) * 128), int32_t(at.row8 * 8),
                         int32_t(at.group), bar, policy);
        if constexpr (nvfp4_weights(KIND))
          ptx::tma_load_2d(ring_scales + place * L::kScaleBytes, &a.scales[matrix], int32_t(at.row8 * 128),
                           int32_t(at.group / 4 * (a.k / 64) + (chunk0 + next_chunk) * 4), bar, policy);
      }
      if (++next_slot == kSlots) next_slot = 0;
      if (PAIR && (next_matrix ^= 1) != 0) return;
      ++next;
      if (++next_chunk == chunks) { next_chunk = 0; ++next_block; }
    };
    // Settled weights do not depend on the kernel before this one (it wrote activations): ask for them while it still runs.
    // Others come as far as L2 meanwhile and are asked for behind the tokens, whose loads would queue behind theirs (MLP of
    // one NVFP4 row, us: settled 49.2, two pieces from L2 50.2, four 51.1, asked for before the tokens 52.0, no prefetch 52.9).
    const bool unsettled = !a.weights_settled && slab_begin == piece_begin;
    if (unsettled) {
#pragma unroll 1
      for (uint32_t s = 0; s < kSlots; ++s) request(true);
      next = begin; next_block = block; next_chunk = chunk; next_slot = turn % kSlots; next_matrix = 0;
    } else {
#pragma unroll 1
      for (uint32_t s = 0; s < kSlots; ++s) request();
    }
    if (slab_begin != piece_begin) __syncthreads();        // everyone is done with the slab before
    const bool ragged = a.k % chunk_values(KIND) != 0;
    if (ragged || (slab_begin == piece_begin && a.rows < NT * 8))      // token columns and values of K that do not exist
      for (uint32_t i = threadIdx.x; i < a.chunks_per_slab * L::kChunkBytes / 16; i += L::kThreads)
        reinterpret_cast<uint4*>(tokens)[i] = make_uint4(0, 0, 0, 0);
    if (slab_begin == piece_begin) griddep_enter();
    __syncthreads();
    stage_tokens<KIND, NT, PAIR>(a, chunk0, chunks, a.packed != nullptr && slab_begin == base, tokens);
    if (unsettled)
#pragma unroll 1
      for (uint32_t s = 0; s < kSlots; ++s) request();
    __syncthreads();

    constexpr int kMatrices = PAIR ? 2 : 1, kSums = lane_sums<NT, PAIR>();
    float acc[kMatrices][2][NT][4] = {};
    const auto sum_at = [&](int i) -> float& { return acc[i / (NT * 8)][i / 4 % 2][i / 8 % NT][i % 4]; };
    float* mine = sums + warp * kValues + lane;
    const auto put = [&](float* to) {
#pragma unroll
      for (int i = 0; i < kSums; ++i) to[i * 32] = sum_at(i);
    };
    bool head = begin_chunk != 0;            // the row block under way was begun by the warp before this one
#pragma unroll 1
    for (uint32_t piece = begin; piece < end; ++piece) {
#pragma unroll
      for (int m = 0; m < kMatrices; ++m, ++turn) {
        const uint32_t place = warp * kSlots + turn % kSlots;
        if (!ptx::mbar_wait_warp(full_bar + place, turn / kSlots & 1u)) {
          if (lane == 0 && a.error != nullptr) atomicCAS(a.error, 0u, 0xA0000000u | (blockIdx.x << 8) | place);
          return;
        }
        uint32_t scale[4] = {};
        if constexpr (nvfp4_weights(KIND)) {
          const uint4 s = ptx::lds128(ptx::smem_u32(ring_scales + place * L::kScaleBytes) + lane % 4 * 128 + lane / 4 * 16);
          scale[0] = s.x; scale[1] = s.y; scale[2] = s.z; scale[3] = s.w;
        }
        const auto multiply_into = [&](float (*sum)[NT][4]) {
          multiply<KIND, NT>(ptx::smem_u32(ring + place * kPieceBytes) + lane / 4 * 128, lane, scale,
                             ptx::smem_u32(tokens) + chunk * L::kChunkBytes, sum);
        };
        if constexpr (PIECE_SUMS) {
          float of_piece[2][NT][4] = {};
          multiply_into(of_piece);
          __syncwarp();                                        // every lane has read the slot
          request();
#pragma unroll
          for (int i = 0; i < 8 * NT; ++i) acc[m][i / 4 % 2][i / 8][i % 4] += of_piece[i / 4 % 2][i / 8][i % 4];
        } else {
          multiply_into(acc[m]);
          __syncwarp();
          request();
        }
      }
      if (++chunk != chunks) continue;
      // the row block ends here
      if (head) {
        put(mine);
      } else {
        Sums<NT, PAIR> sum;
#pragma unroll
        for (int i = 0; i < kSums; ++i) sum.v[i] = sum_at(i);
        finish_unit<NT, PAIR>(a, slab.slab * a.blocks + block, unit_first, a.slabs == 1, lane, sum);
      }
      head = false;
      chunk = 0;
      ++block;
#pragma unroll
      for (int i = 0; i < kSums; ++i) sum_at(i) = 0.0F;
    }
    if (head && chunk != begin_chunk) put(mine);            // it ends in a later warp
    const bool tail = !head && chunk != 0;                  // begun here, ends in a later warp
    __syncthreads();
    // ---- row blocks that several warps share: the warp with the first part adds the others' to it, in order.  That is
    // the one that began the row block, or warp 0 when another SM did.
#pragma unroll 1
    for (uint32_t pass = 0; pass < 2; ++pass) {
      if (pass == 0 ? warp != 0 || begin_chunk == 0 : !tail) continue;
      const uint32_t shared_block = block_of(a, slab.slab, (pass == 0 ? begin : end - 1) - base);
      const uint32_t unit_begin = base + shared_block * chunks, unit_end = unit_begin + chunks;
      Sums<NT, PAIR> sum;
#pragma unroll
      for (int i = 0; i < kSums; ++i) sum.v[i] = pass == 0 ? mine[i * 32] : sum_at(i);
#pragma unroll 1
      for (uint32_t w = warp + 1; w < kWarps && warp_begin(w) < unit_end; ++w) {
        if (warp_begin(w) == warp_begin(w + 1)) continue;
        const float* theirs = sums + w * kValues + lane;
#pragma unroll
        for (int i = 0; i < kSums; ++i) sum.v[i] += theirs[i * 32];
      }
      finish_unit<NT, PAIR>(a, slab.slab * a.blocks + shared_block, unit_first,
                            a.slabs == 1 && unit_begin >= slab_begin && unit_end <= slab_end, lane, sum);
    }
    slab_unit = (slab.slab + 1) * a.blocks;
    slab_begin = slab_end;
  }
}

template <StreamKind KIND, int NT, bool PAIR, bool PIECE_SUMS>
cudaError_t launch_instance(const StreamArgs& args, const StreamPlan& plan, cudaStream_t stream) {
  static bool configured_on[kMaxDeviceSlots] = {};   // the attribute is per GPU
  bool& configured = configured_on[current_device_slot()];
  if (!configured) {
    const cudaError_t status = cudaFuncSetAttribute(decode_stream_kernel<KIND, NT, PAIR, PIECE_SUMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedLimit);
    if (status != cudaSuccess) return status;
    configured = true;
  }
  return launch_pdl_shared(decode_stream_kernel<KIND, NT, PAIR, PIECE_SUMS>, plan.grid, Layout<KIND, NT, PAIR>::kThreads, plan.shared_bytes, stream, args);
}

template <StreamKind KIND>
cudaError_t launch_kind(const StreamArgs& args, const StreamPlan& plan, bool pair, cudaStream_t stream) {
  if constexpr (KIND == StreamKind::w4a16) {
    if (plan.tiles == 2) return pair ? launch_instance<KIND, 2, true, false>(args, plan, stream) : launch_instance<KIND, 2, false, false>(args, plan, stream);
  } else if (plan.piece_sums) {
    return pair ? launch_instance<KIND, 1, true, true>(args, plan, stream) : launch_instance<KIND, 1, false, true>(args, plan, stream);
  }
  return pair ? launch_instance<KIND, 1, true, false>(args, plan, stream) : launch_instance<KIND, 1, false, false>(args, plan, stream);
}

struct Sizes { uint32_t warps, fixed, chunk; };
template <StreamKind KIND>
Sizes sizes_of(bool two, bool pair) {
  const auto of = [](auto layout) { using L = decltype(layout); return Sizes{L::kWarps, L::kFixedBytes, L::kChunkBytes}; };
  if constexpr (KIND == StreamKind::w4a16)
    if (two) return pair ? of(Layout<KIND, 2, true>{}) : of(Layout<KIND, 2, false>{});
  return pair ? of(Layout<KIND, 1, true>{}) : of(Layout<KIND, 1, false>{});
}

uint32_t row_bytes_of(StreamKind kind, uint32_t k) { return nvfp4_weights(kind) ? k / 2 : kind == StreamKind::w8a8 ? k : 2 * k; }

}  // namespace

StreamPlan plan_stream(StreamKind kind, uint32_t rows, uint32_t k, uint32_t n, bool pair, int sm_count) {
  StreamPlan p;
  const bool nvfp4 = nvfp4_weights(kind);
  // rows come in groups of 32 (the tensor map must not reach past the matrix), tokens in groups of sixteen values
  if (rows == 0 || rows > kStreamMaxRows || k % (nvfp4 ? 64 : 16) != 0 || n % 32 != 0 || n == 0 || k == 0) return p;
  // A second group of eight tokens costs half as many instructions again per weight byte; where another kernel runs the same
  // projection, it is the faster one from nine rows on.
  if (rows > 8 && kind != StreamKind::w4a16) return p;
  p.physical_n = n;
  p.tiles = rows <= 8 ? 1 : 2;
  p.blocks = int((n + 127) / 128 * 4);
  p.chunks = int((k + chunk_values(kind) - 1) / chunk_values(kind));
  const Sizes size = kind == StreamKind::w4a4    ? sizes_of<StreamKind::w4a4>(p.tiles == 2, pair)
                     : kind == StreamKind::w4a16 ? sizes_of<StreamKind::w4a16>(p.tiles == 2, pair)
                     : kind == StreamKind::w8a8  ? sizes_of<StreamKind::w8a8>(p.tiles == 2, pair)
                                                 : sizes_of<StreamKind::w16a16>(p.tiles == 2, pair);
  const int most = int((kSharedLimit - size.fixed) / size.chunk);
  p.slabs = (p.chunks + most - 1) / most;
  p.chunks_per_slab = (p.chunks + p.slabs - 1) / p.slabs;
  p.slabs = (p.chunks + p.chunks_per_slab - 1) / p.chunks_per_slab;
  const uint64_t pieces = uint64_t(p.blocks) * p.chunks;
  if (pieces >= (1u << 30) || p.slabs > 32) return p;          // one lane per slab when the sums are added
  // Whole row blocks for every SM, where all of K fits: the sums of a block that SMs share cost a pass through L2, 2 us, more than
  // some SMs with one block more than others do.  (Shared / whole, us: NVFP4 1x2816x2048 7.3 / 5.0, 1x2816x8192 9.1 / 6.9, 1x5376x21504
  // 17.3 / 15.2, FP8 8x2816x4096 9.7 / 6.6, 4x5376x43008 38.6 / 36.4, BF16 8x2816x1024 7.9 / 6.1.)  Blocks of a short K come together
  // until they feed a block's warps; an SM for each is the slower way (NVFP4 1x1024x4864 4.8 / 5.4, FP8 1x512x4864 3.7 / 4.3).
  const auto share = [](uint64_t all, uint64_t of) { return (all + of - 1) / of; };
  const bool one_each = p.blocks <= sm_count && 2 * p.blocks >= sm_count;
  const int together = std::max(1, int(size.warps) / p.chunks);
  const int whole_grid = one_each ? p.blocks : int(std::min<uint64_t>(sm_count, share(p.blocks, together)));
  const int cut_grid = int(std::min<uint64_t>(sm_count, share(pieces, size.warps)));          // at least one piece per warp
  const bool cuts = p.chunks_per_slab / int(pieces / cut_grid) + 2 <= 32;                     // one lane per part of a slab's row block
  // Where a warp has more pieces than with equal ranges its sums would be longer, and further from the exact ones: each piece is
  // then summed by itself, for 0.5 to 3 % of the time (outputs that are not the nearest BF16, shared / whole / whole with sums of pieces:
  // BF16 1x5376x1024 9.8e-5 / 2.8e-4 / 9.8e-5, 4x5376x2048 1.6e-4 / 3.4e-4 / 1.4e-4).  W4A16, whose time goes into decoding, stays
  // shared there (MLP of one row, whole / shared, us: 5376 -> 4864 26.5 / 23.8, 5376 -> 14336 48.1 / 46.5, 5376 -> 21504 61.4 / 61.8;
  // but 2816 -> 6144, as many pieces, 17.2 / 20.2).
  const bool longer = !one_each && share(share(p.blocks, whole_grid) * p.chunks, size.warps) > share(share(pieces, cut_grid), size.warps);
  p.whole = p.slabs == 1 && (kind != StreamKind::w4a16 || !longer || !cuts);
  p.piece_sums = p.whole && longer && kind != StreamKind::w4a16;
  if (!p.whole && !cuts) return p;
  p.grid = p.whole ? whole_grid : cut_grid;
  const int per_cta = int(pieces / p.grid);
  const int shortest = p.chunks - (p.slabs - 1) * p.chunks_per_slab;
  p.max_units = per_cta / shortest + 3;
  p.shared_bytes = size_t(p.chunks_per_slab) * size.chunk + size.fixed;
  if (!p.whole) {
    p.workspace_bytes = size_t(p.grid) * p.max_units * p.tiles * (pair ? 512 : 256) * sizeof(float);
    p.counter_count = size_t(p.blocks);
  }
  p.usable = p.workspace_bytes <= (size_t(16) << 20);          // callers size their scratch by upper bounds above this
  return p;
}

bool StreamMaps::get(StreamKind kind, const StreamMatrix& m, uint32_t n, uint32_t k, std::string* error) {
  if (m.data != data) {
    if (!encode_tensor_map_piece(&weights, m.data, row_bytes_of(kind, k), n, error)) return false;
    data = m.data;
  }
  if (nvfp4_weights(kind) && m.scales != scale_data) {
    if (!encode_tensor_map_atoms(&scales, m.scales, uint64_t((n + 127) / 128) * ((k + 63) / 64), error)) return false;
    scale_data = m.scales;
  }
  return true;
}

bool stream_aligned(const StreamProblem& q) {
  const auto off = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16; };
  return !off(q.input) && !off(q.first.data) && !off(q.second.data) && !off(q.first.scales) && !off(q.second.scales);
}

cudaError_t launch_stream(const StreamProblem& q, const StreamPlan& plan, const StreamMaps& first, const StreamMaps& second,
                          cudaStream_t stream) {
  StreamArgs a{};
  const StreamMatrix* matrix[2] = {&q.first, &q.second};
  const StreamMaps* maps[2] = {&first, &second};
  const bool pair = q.second.data != nullptr;
  for (int i = 0; i < (pair ? 2 : 1); ++i) {
    a.weights[i] = maps[i]->weights;
    a.scales[i] = maps[i]->scales;
    a.alpha[i] = matrix[i]->alpha * (q.kind == StreamKind::w4a16 ? kW4a16Alpha : 1.0F);
    a.channel_alpha[i] = matrix[i]->channel_alpha;
  }
  a.input = static_cast<const bf16*>(q.input);
  a.out = static_cast<bf16*>(q.output);
  a.ld_out = q.ld_out;
  a.partials = static_cast<float*>(q.workspace);
  a.counters = q.counters;
  a.packed = q.packed;
  a.packed_scales = q.packed_scales;
  a.error = q.error;
  a.reread = q.reread ? 1 : 0;
  a.weights_settled = q.weights_settled ? 1 : 0;
  a.inverse_scale = q.inverse_scale;
  a.rows = q.rows;
  a.k = q.k;
  a.n = q.n;
  a.gelu = q.gelu ? 1 : 0;
  a.blocks = uint32_t(plan.blocks);
  a.chunks = uint32_t(plan.chunks);
  a.chunks_per_slab = uint32_t(plan.chunks_per_slab);
  a.slabs = uint32_t(plan.slabs);
  a.max_units = uint32_t(plan.max_units);
  const uint32_t steps = plan.whole ? a.blocks : a.blocks * a.chunks;
  a.step = plan.whole ? a.chunks : 1;
  a.range = steps / uint32_t(plan.grid);
  a.longer = steps % uint32_t(plan.grid);
  a.by_range = Divisor::of(a.range);
  a.by_range1 = Divisor::of(a.range + 1);
  a.by_slab = Divisor::of(a.blocks * a.chunks_per_slab);
  a.by_chunks = Divisor::of(a.chunks_per_slab);
  a.by_last_chunks = Divisor::of(a.chunks - (a.slabs - 1) * a.chunks_per_slab);
  a.by_blocks = Divisor::of(a.blocks);
  switch (q.kind) {
    case StreamKind::w4a4: return launch_kind<StreamKind::w4a4>(a, plan, pair, stream);
    case StreamKind::w4a16: return launch_kind<StreamKind::w4a16>(a, plan, pair, stream);
    case StreamKind::w8a8: return launch_kind<StreamKind::w8a8>(a, plan, pair, stream);
    case StreamKind::w16a16: return launch_kind<StreamKind::w16a16>(a, plan, pair, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gw
