// Work of the grouped NVFP4 GEMMs of the MoE layer, found on the device: every CTA turns the expert offsets into a
// table of (first row, row count, first work unit) per expert.  Offsets beyond the declared capacity are clamped and
// reported.
#pragma once

#include "gemm_pair_moe.h"

namespace gw::moe_work {

constexpr int kExperts = 128;

struct WorkTable {
  int32_t first[kExperts];        // first sorted row of the expert (clamped to the capacity)
  int32_t count[kExperts];        // its rows
  int32_t prefix[kExperts + 1];   // first work unit of the expert; [128] = all units
};

struct Unit {
  int e, first, count;
  int tile;      // token tile inside the expert
  int part;      // channel tile or chunk of channels
};

// All threads of the CTA.  units_per_tile work units for every token tile (ROWS rows) of every expert whose projections
// FIRST .. LAST (0 gate, 1 up, 2 down) run as the launch's kind; rows of an expert that lives on another GPU get no work.
template <int ROWS, int FIRST, int LAST>
__device__ __forceinline__ void build_work_table(const PairMoeParams& p, WorkTable* t, int units_per_tile) {
  __shared__ int32_t warp_totals[4];
  const int e = threadIdx.x;
  int32_t units = 0;
  if (e < kExperts) {
    int32_t first = p.offsets[e], last = p.offsets[e + 1];
    const bool here = moe_effective_kind(p.experts[e].storage[FIRST], p.fp4) == p.kind &&
                      moe_effective_kind(p.experts[e].storage[LAST], p.fp4) == p.kind;
    const int32_t capacity = int32_t(p.capacity);
    if (first < 0 || last < first || last > capacity) {
      if (p.error != nullptr) atomicCAS(p.error, 0u, 0x70000100u | uint32_t(e));
      first = min(max(first, 0), capacity);
      last = min(max(last, first), capacity);
    }
    t->first[e] = first;
    t->count[e] = last - first;
    units = here ? ((last - first + ROWS - 1) / ROWS) * units_per_tile : 0;
  }
  // exclusive scan over the 128 experts: shuffles inside each of the first four warps, then their totals
  int32_t scan = units;
  const int lane = threadIdx.x % 32;
  if (e < kExperts) {
#pragma unroll
    for (int step = 1; step < 32; step *= 2) {
      const int32_t other = __shfl_up_sync(0xffffffffu, scan, step);
      if (lane >= step) scan += other;
    }
    if (lane == 31) warp_totals[e / 32] = scan;
  }
  __syncthreads();
  if (e < kExperts) {
    int32_t base = 0;
    for (int w = 0; w < e / 32; ++w) base += warp_totals[w];
    t->prefix[e] = base + scan - units;
    if (e == kExperts - 1) t->prefix[kExperts] = base + scan;
  }
  __syncthreads();
}

__device__ __forceinline__ void decode_unit(const WorkTable* t, int w, int units_per_tile, Unit& u) {
  if (u.e < 0 || w < t->prefix[u.e] || w >= t->prefix[u.e + 1]) {
    int lo = 0, hi = kExperts;             // largest e with prefix[e] <= w (it has units, since w < prefix[128])
    while (lo + 1 < hi) {
      const int mid = (lo + hi) / 2;
      if (t->prefix[mid] <= w) lo = mid; else hi = mid;
    }
    u.e = lo;
    u.first = t->first[lo];
    u.count = t->count[lo];
  }
  const int local = w - t->prefix[u.e];
  u.part = local % units_per_tile;
  u.tile = local / units_per_tile;
}

// The same with the token tiles of an expert fastest, so that the second one under a channel tile finds the weights in L2.
// Returns the expert's token tiles.
template <int ROWS>
__device__ __forceinline__ int place_unit(const WorkTable* t, int w, int units_per_tile, Unit& u) {
  decode_unit(t, w, units_per_tile, u);
  const int local = u.tile * units_per_tile + u.part, tiles = (u.count + ROWS - 1) / ROWS;
  u.part = local / tiles;
  u.tile = local - u.part * tiles;
  return tiles;
}

// This CTA's contiguous share of the units.
struct Range { int begin, end; };
__device__ __forceinline__ Range my_range(int total) {
  return {int((long long)(total) * blockIdx.x / gridDim.x), int((long long)(total) * (blockIdx.x + 1) / gridDim.x)};
}
// Token columns of a tile that hold rows of the expert, and the MMA's N.
__device__ __forceinline__ int valid_columns(const Unit& u, int tile_rows) { return min(tile_rows, u.count - u.tile * tile_rows); }
__device__ __forceinline__ int mma_columns(int valid) { return (valid + 15) & ~15; }

// ---- epilogue warps of the kernels with an expert's tokens on the columns
// A tile of 128 tokens keeps sixteen epilogue warps busy; with 64 the wider launch costs more than it gives (MoE layer of
// 64 tokens, us, 8 / 16 warps: 81.7 / 86.5; 1500 tokens with popular experts on 128-wide tiles 181 / 170).
template <int TILE> constexpr int kEpilogueWarps = TILE == 128 ? 16 : 8;
template <int THREADS>
__device__ __forceinline__ void epilogue_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }
// The same with a vote: every epilogue thread learns whether one of them gave up, so that all of them leave together.
template <int THREADS>
__device__ __forceinline__ bool epilogue_barrier_any(bool failed) {
  uint32_t any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(any) : "r"(uint32_t(failed)), "n"(THREADS) : "memory");
  return any != 0;
}

}  // namespace gw::moe_work
