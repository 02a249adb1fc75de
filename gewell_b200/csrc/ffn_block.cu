// The feed-forward block of one Gemma-4-26B-A4B layer around the MoE, behind
// the C ABI: the three-output RMS norm that feeds the shared MLP, the router
// and the experts, the shared MLP, the router projection, the MoE layer, the
// three post norms with their residual adds and the layer scalar -- the second
// half of BatchedExecutor's layer loop in the reference
// (models/gemma4/26b_a4b/sm120/batched_executor.cu:250-286) with the element-wise
// math of bf16_math.cuh:17-117.
//
// Every BF16 rounding of the reference is kept, and so is the order of its
// FP32 row reduction (the reference builds without fused multiply-add and
// fixes the order to match a pinned FP32 mean): element i of a row belongs to
// logical lane (i / 4) % lanes and accumulator i % 4, an accumulator adds its
// squares by ascending i, a lane's total is ((a0 + a1) + a2) + a3, and lanes
// fold in a halving tree.  `lanes` depends on the row count and the width.
//
// Here a row is read from HBM once: every thread keeps its eight (or 16, 32) values and their weights in
// registers between the reduction and the output, and the row sits in shared memory for the fixed-order sums
// only.  What bounds these kernels at decode sizes is the chain of memory latency, barriers and adds, not
// bytes: all loads of a thread are 16 bytes wide and issued before the first barrier (2816 wide, 8 rows, weights
// not in L2, launches of a graph behind one another: norm 4.5 -> 2.2 us, three outputs 8.6 -> 2.7, tail 9.6 -> 4.1 us, against
// element-wise loads in the output loop and a block barrier for every level of the sum).  The block's tail -- two post norms, add, the third norm, residual
// add, layer scalar: seven launches in the reference -- is one kernel with one block per row.
#include <algorithm>
#include <cmath>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "combine.cuh"
#include "common.cuh"
#include "dense.h"
#include "kernels.h"
#include "moe_kernels.h"

using namespace gw;

namespace {

constexpr int kNormThreads = 512;                // at most; a block has a thread for every eight values of a row
constexpr float kRmsEpsilon = 1e-6F;   // include/gewell/models/gemma4/26b_a4b/model.h:26

uint32_t floor_power_of_two(uint32_t value) {
  uint32_t result = 1;
  while (result * 2 <= value) result *= 2;
  return result;
}

// Logical lanes of the row reduction for a launch of `rows` rows of `width` values: the rule of
// normalize_to (bf16_math.cuh:86-95) -- as many lanes as the width feeds with whole 4-vectors, at most
// 512, shared among up to 16 rows.
uint32_t reduction_lanes(uint32_t rows, uint32_t width) {
  const uint32_t by_width = floor_power_of_two(std::min<uint32_t>(512, std::max<uint32_t>(1, width / 4)));
  const uint32_t by_rows = 512 / floor_power_of_two(std::min<uint32_t>(16, std::max<uint32_t>(1, rows)));
  return std::min(by_width, by_rows);
}

__device__ __forceinline__ float as_float(bf16 v) { return __bfloat162float(v); }
__device__ __forceinline__ bf16 rounded(float v) { return __float2bfloat16_rn(v); }

// Eight BF16 values as a thread loads and keeps them; thread t has vectors t, t + blockDim.x, ... of a row.
union Vec {
  uint4 bits;
  bf16 v[8];
};
template <int NV>
struct RowPart {
  Vec part[NV];
  __device__ __forceinline__ void load(const bf16* __restrict__ row, uint32_t vectors) {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const uint32_t i = threadIdx.x + j * blockDim.x;
      part[j].bits = i < vectors ? *(reinterpret_cast<const uint4*>(row) + i) : make_uint4(0, 0, 0, 0);
    }
  }
  // 16-bit loads for a row that is not 16-byte aligned (a weight vector inside a larger buffer)
  __device__ __forceinline__ void load_any(const bf16* __restrict__ row, uint32_t vectors) {
    if (reinterpret_cast<uintptr_t>(row) % 16 == 0) return load(row, vectors);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const uint32_t i = threadIdx.x + j * blockDim.x;
      part[j].bits = make_uint4(0, 0, 0, 0);
      if (i < vectors)
#pragma unroll
        for (int e = 0; e < 8; ++e) part[j].v[e] = row[size_t(i) * 8 + e];
    }
  }
  __device__ __forceinline__ void store(bf16* row, uint32_t vectors) const {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const uint32_t i = threadIdx.x + j * blockDim.x;
      if (i < vectors) *(reinterpret_cast<uint4*>(row) + i) = part[j].bits;
    }
  }
  __device__ __forceinline__ void store_any(bf16* row, uint32_t vectors) const {
    if (reinterpret_cast<uintptr_t>(row) % 16 == 0) return store(row, vectors);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const uint32_t i = threadIdx.x + j * blockDim.x;
      if (i < vectors)
#pragma unroll
        for (int e = 0; e < 8; ++e) row[size_t(i) * 8 + e] = part[j].v[e];
    }
  }
};

struct NormArgs {
  const bf16* input;
  uint32_t width, lanes;
  float inverse_width;
};

// 1 / sqrt(mean(row^2) + eps) of ROWS rows in shared memory, in the reference's order (see the head of this file).
// A thread takes whole logical lanes (four accumulators, eight bytes a step); warp r folds the lane totals of row r,
// the levels inside a warp by shuffles.  `totals` holds ROWS * lanes floats.  Every thread gets the results.  No
// fused multiply-add anywhere: the reference's translation unit is built with --fmad=false.
template <int ROWS>
__device__ __forceinline__ void inverse_rms(const NormArgs& a, const bf16* const (&rows)[ROWS], float* totals, float (&inverse)[ROWS]) {
  __shared__ float result[ROWS];
  __syncthreads();                                     // the rows are complete; `totals` is free
  const uint32_t lanes = a.lanes;                      // a power of two; 4 * lanes <= width
  if (lanes >= 8 && lanes <= 64) {
    // Launches of many rows have few logical lanes, which walk far: a thread per accumulator, so that 32 lanes keep 128 threads
    // busy (feed-forward block of 4000 rows, with three blocks of the tail an SM: 403 -> 369 us).
    const uint32_t shift = 31 - __clz(4 * lanes);
    for (uint32_t item = threadIdx.x; item < ROWS * 4 * lanes; item += blockDim.x) {      // whole warps
      const uint32_t which = ROWS == 1 ? 0 : item >> shift, l = item & (4 * lanes - 1);
      const bf16* row = rows[0];
#pragma unroll
      for (int r = 1; r < ROWS; ++r)
        if (which == uint32_t(r)) row = rows[r];
      float sum = 0.F;
#pragma unroll 4
      for (uint32_t i = l; i < a.width; i += 4 * lanes) {
        const float v = as_float(row[i]);
        sum = __fadd_rn(sum, __fmul_rn(v, v));
      }
      float total = __fadd_rn(sum, __shfl_down_sync(0xffffffffu, sum, 1));
      total = __fadd_rn(total, __shfl_down_sync(0xffffffffu, sum, 2));
      total = __fadd_rn(total, __shfl_down_sync(0xffffffffu, sum, 3));
      if (l % 4 == 0) totals[item / 4] = total;
    }
  } else {
    for (uint32_t item = threadIdx.x; item < ROWS * lanes; item += blockDim.x) {
      const uint32_t which = ROWS == 1 ? 0 : item / lanes, l = ROWS == 1 ? item : item % lanes;
      const bf16* row = rows[0];
#pragma unroll
      for (int r = 1; r < ROWS; ++r)
        if (which == r) row = rows[r];
      float sum[4] = {0.F, 0.F, 0.F, 0.F};
#pragma unroll 4
      for (uint32_t i = 4 * l; i < a.width; i += 4 * lanes) {
        const uint2 bits = *reinterpret_cast<const uint2*>(row + i);
        const float v[4] = {bf16_bits_to_float(bits.x & 0xffff), bf16_bits_to_float(bits.x >> 16), bf16_bits_to_float(bits.y & 0xffff),
                            bf16_bits_to_float(bits.y >> 16)};
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] = __fadd_rn(sum[e], __fmul_rn(v[e], v[e]));
      }
      totals[item] = __fadd_rn(__fadd_rn(__fadd_rn(sum[0], sum[1]), sum[2]), sum[3]);
    }
  }
  __syncthreads();
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32, warps = blockDim.x / 32;
  for (uint32_t r = warp; r < uint32_t(ROWS); r += warps) {
    float* mine = totals + r * lanes;
    for (uint32_t stride = lanes / 2; stride >= 32; stride /= 2) {
      for (uint32_t l = lane; l < stride; l += 32) mine[l] = __fadd_rn(mine[l], mine[l + stride]);
      __syncwarp();
    }
    float sum = lane < lanes ? mine[lane] : 0.F;
    for (uint32_t stride = (lanes < 32 ? lanes : 32) / 2; stride; stride /= 2)
      sum = __fadd_rn(sum, __shfl_down_sync(0xffffffffu, sum, stride));
    if (lane == 0) result[r] = rsqrtf(__fadd_rn(__fmul_rn(sum, a.inverse_width), kRmsEpsilon));
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ROWS; ++r) inverse[r] = result[r];
}

// y = bf16(x * inv * w)   (w == nullptr: no weight)       -- NormOutput, bf16_math.cuh:18-24
template <int NV>
__global__ void __launch_bounds__(kNormThreads) rms_norm_kernel(NormArgs a, const bf16* __restrict__ weight, bf16* __restrict__ output) {
  extern __shared__ __align__(16) unsigned char norm_smem[];
  bf16* row = reinterpret_cast<bf16*>(norm_smem);
  float* totals = reinterpret_cast<float*>(norm_smem + size_t(a.width) * sizeof(bf16));
  const uint32_t vectors = a.width / 8;
  griddep_enter();
  RowPart<NV> x, w;
  x.load(a.input + size_t(blockIdx.x) * a.width, vectors);
  if (weight) w.load_any(weight, vectors);
  x.store(row, vectors);
  float inv[1];
  inverse_rms<1>(a, {row}, totals, inv);
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float v = __fmul_rn(as_float(x.part[j].v[e]), inv[0]);
      x.part[j].v[e] = rounded(weight ? __fmul_rn(v, as_float(w.part[j].v[e])) : v);
    }
  x.store_any(output + size_t(blockIdx.x) * a.width, vectors);
}

struct FeedForwardNormArgs {
  const bf16 *shared_weight, *router_weight, *expert_weight;
  bf16 *shared, *router, *expert;
  float router_scale;                    // 1 / sqrt(width), formed on the host
};

// FeedForwardNormOutput (bf16_math.cuh:25-37): one RMS, three outputs; the router input keeps its three
// separate roundings (unweighted norm, weighted product, final scale).
template <int NV>
__global__ void __launch_bounds__(kNormThreads) rms_norm_feedforward_kernel(NormArgs a, FeedForwardNormArgs f) {
  extern __shared__ __align__(16) unsigned char norm_smem[];
  bf16* row = reinterpret_cast<bf16*>(norm_smem);
  float* totals = reinterpret_cast<float*>(norm_smem + size_t(a.width) * sizeof(bf16));
  const uint32_t vectors = a.width / 8;
  griddep_enter();
  RowPart<NV> x, shared, expert, router;
  x.load(a.input + size_t(blockIdx.x) * a.width, vectors);
  shared.load_any(f.shared_weight, vectors);
  expert.load_any(f.expert_weight, vectors);
  router.load_any(f.router_weight, vectors);
  x.store(row, vectors);
  float inv[1];
  inverse_rms<1>(a, {row}, totals, inv);
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float v = __fmul_rn(as_float(x.part[j].v[e]), inv[0]);
      shared.part[j].v[e] = rounded(__fmul_rn(v, as_float(shared.part[j].v[e])));
      expert.part[j].v[e] = rounded(__fmul_rn(v, as_float(expert.part[j].v[e])));
      const bf16 weighted = rounded(__fmul_rn(as_float(rounded(v)), as_float(router.part[j].v[e])));
      router.part[j].v[e] = rounded(__fmul_rn(as_float(weighted), f.router_scale));
    }
  const size_t base = size_t(blockIdx.x) * a.width;
  shared.store_any(f.shared + base, vectors);
  expert.store_any(f.expert + base, vectors);
  router.store_any(f.router + base, vectors);
}

struct TailArgs {
  const bf16* shared_mlp;                             // [rows, width]: shared MLP output
  bf16* routed;                                       // MoE output
  const bf16 *norm_shared, *norm_routed, *norm_sum;   // post_feedforward_norm_1, _2, post_feedforward_norm
  const bf16* layer_scalar;                           // [1]
  bf16* hidden;                                       // [rows, width], updated in place
  // COMBINE: `routed` is this kernel's output as well, the weighted sum of the token's eight expert rows
  const uint4* down;
  const int32_t* inverse;
  const float* weights;
};
constexpr int kTopK = 8;
constexpr int kBlockThreads = 2816 / 8;     // COMBINE: of the block's own width.  Three of its launch's blocks fit an SM (56 registers, not 63)

// shared = norm1(shared_mlp); branch = norm2(routed); sum = bf16(shared + branch); branch = norm3(sum);
// hidden = bf16(hidden + branch); hidden = bf16(hidden * scalar)        (batched_executor.cu:260,278-285)
// (A bound of one block an SM instead of none makes the others 80 registers of 63 and spill more: 4096 rows of 4096 values 82 -> 143 us.)
template <int NV, bool COMBINE>
__global__ void __launch_bounds__((COMBINE ? kBlockThreads : kNormThreads), (COMBINE ? 3 : 0)) ffn_tail_kernel(NormArgs a, TailArgs t) {
  static_assert(!COMBINE || NV == 1, "one vector a thread");
  extern __shared__ __align__(16) unsigned char norm_smem[];
  bf16* first = reinterpret_cast<bf16*>(norm_smem);
  bf16* second = first + a.width;
  float* totals = reinterpret_cast<float*>(norm_smem + size_t(2) * a.width * sizeof(bf16));
  const size_t base = size_t(blockIdx.x) * a.width;
  const uint32_t vectors = a.width / 8;
  // inside a block the launch before is the experts' down GEMM, which writes none of the four weights below
  if constexpr (!COMBINE) griddep_enter();
  RowPart<NV> shared, branch, norm_shared, norm_routed, norm_sum, hidden;
  norm_shared.load_any(t.norm_shared, vectors);
  norm_routed.load_any(t.norm_routed, vectors);
  norm_sum.load_any(t.norm_sum, vectors);
  const float scalar = as_float(*t.layer_scalar);
  if constexpr (COMBINE) griddep_enter();
  shared.load(t.shared_mlp + base, vectors);
  if constexpr (COMBINE) {
    __shared__ int32_t slot_row[kTopK];
    __shared__ float slot_weight[kTopK];
    if (threadIdx.x < kTopK) {
      slot_row[threadIdx.x] = t.inverse[size_t(blockIdx.x) * kTopK + threadIdx.x];
      slot_weight[threadIdx.x] = t.weights[size_t(blockIdx.x) * kTopK + threadIdx.x];
    }
    __syncthreads();
    branch.part[0].bits = make_uint4(0, 0, 0, 0);
    if (threadIdx.x < vectors) branch.part[0].bits = combine_rows<kTopK>(t.down, slot_row, slot_weight, vectors, threadIdx.x);
    branch.store(t.routed + base, vectors);
  } else {
    branch.load(t.routed + base, vectors);
  }
  hidden.load_any(t.hidden + base, vectors);
  shared.store(first, vectors);
  branch.store(second, vectors);
  float inv[2], inv_sum[1];
  inverse_rms<2>(a, {first, second}, totals, inv);
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const bf16 x = rounded(__fmul_rn(__fmul_rn(as_float(shared.part[j].v[e]), inv[0]), as_float(norm_shared.part[j].v[e])));
      const bf16 y = rounded(__fmul_rn(__fmul_rn(as_float(branch.part[j].v[e]), inv[1]), as_float(norm_routed.part[j].v[e])));
      shared.part[j].v[e] = rounded(__fadd_rn(as_float(x), as_float(y)));
    }
  shared.store(first, vectors);
  inverse_rms<1>(a, {first}, totals, inv_sum);
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const bf16 x = rounded(__fmul_rn(__fmul_rn(as_float(shared.part[j].v[e]), inv_sum[0]), as_float(norm_sum.part[j].v[e])));
      const bf16 updated = rounded(__fadd_rn(as_float(hidden.part[j].v[e]), as_float(x)));
      hidden.part[j].v[e] = rounded(__fmul_rn(as_float(updated), scalar));
    }
  hidden.store_any(t.hidden + base, vectors);
}

// Router logits of few rows: bf16(x . Wrouter^T) for 128 experts.  What bounds it is latency, 720 KB and two to eight
// microseconds of dependent steps; so a block takes sixteen experts and eight rows over all of K, its weights are on their way
// before the wait, every load of a thread is in flight at once and nothing passes through global memory but the
// logits.  (8 rows, alone: weight-streaming kernel 8.7 us, this 4.8.)
// mma.sync: sixteen experts are no tcgen05 tile, and the tensor pipe is idle.  A K step takes any values as long as both
// operands agree: lane 4 * g + t has the same eight consecutive values of expert g, expert g + 8 and row g.
constexpr int kRouterThreads = 256, kRouterSteps = 2816 / 32 / (kRouterThreads / 32);     // of 32 values, each warp
static_assert(kRouterSteps * 32 * (kRouterThreads / 32) == 2816, "whole steps for every warp");
constexpr uint32_t kRouterRows = 128, kRouterExperts = 128;
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__global__ void __launch_bounds__(kRouterThreads)
router_logits_kernel(const uint4* __restrict__ input, const uint4* __restrict__ weights, bf16* __restrict__ logits, uint32_t rows) {
  constexpr uint32_t kVectors = 2816 / 8;
  __shared__ float sums[kRouterThreads / 32][16][8];
  const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x % 32, g = lane / 4, t = lane % 4;
  const uint32_t first = warp * kRouterSteps * 4 + t, expert = blockIdx.x * 16, row = blockIdx.y * 8 + g;
  uint4 lo[kRouterSteps], hi[kRouterSteps], x[kRouterSteps];
#pragma unroll
  for (int i = 0; i < kRouterSteps; ++i) {
    lo[i] = weights[size_t(expert + g) * kVectors + first + 4 * i];
    hi[i] = weights[size_t(expert + g + 8) * kVectors + first + 4 * i];
  }
  griddep_enter();
#pragma unroll
  for (int i = 0; i < kRouterSteps; ++i)
    x[i] = row < rows ? input[size_t(row) * kVectors + first + 4 * i] : make_uint4(0, 0, 0, 0);
  float even[4] = {0.F, 0.F, 0.F, 0.F}, odd[4] = {0.F, 0.F, 0.F, 0.F};
#pragma unroll
  for (int i = 0; i < kRouterSteps; ++i) {
    mma_bf16(even, lo[i].x, hi[i].x, lo[i].y, hi[i].y, x[i].x, x[i].y);
    mma_bf16(odd, lo[i].z, hi[i].z, lo[i].w, hi[i].w, x[i].z, x[i].w);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) sums[warp][g + 8 * (j / 2)][2 * t + j % 2] = even[j] + odd[j];
  __syncthreads();
  const uint32_t e = threadIdx.x % 16, r = threadIdx.x / 16;
  if (r >= 8 || blockIdx.y * 8 + r >= rows) return;
  float sum = 0.F;
#pragma unroll
  for (int w = 0; w < kRouterThreads / 32; ++w) sum += sums[w][e][r];
  logits[size_t(blockIdx.y * 8 + r) * kRouterExperts + expert + e] = rounded(sum);
}

// y = bf16(a + b)                                                       (bf16_math.cuh:109-112)
// VECTOR: every buffer 16-byte aligned, a thread has eight values
template <bool VECTOR>
__global__ void add_kernel(const bf16* a, const bf16* b, bf16* y, size_t n) {
  griddep_enter();
  const size_t i = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) * (VECTOR ? 8 : 1);
  if (VECTOR && i + 8 <= n) {
    Vec u, v;
    u.bits = *reinterpret_cast<const uint4*>(a + i);
    v.bits = *reinterpret_cast<const uint4*>(b + i);
#pragma unroll
    for (int e = 0; e < 8; ++e) u.v[e] = rounded(__fadd_rn(as_float(u.v[e]), as_float(v.v[e])));
    *reinterpret_cast<uint4*>(y + i) = u.bits;
  } else {
    for (size_t j = i; j < n && j < i + (VECTOR ? 8 : 1); ++j) y[j] = rounded(__fadd_rn(as_float(a[j]), as_float(b[j])));
  }
}

// x = bf16(x * scalar[0])                                               (batched_executor.cu:30-33)
template <bool VECTOR>
__global__ void scale_kernel(bf16* x, const bf16* scalar, size_t n) {
  griddep_enter();
  const float s = as_float(*scalar);
  const size_t i = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) * (VECTOR ? 8 : 1);
  if (VECTOR && i + 8 <= n) {
    Vec u;
    u.bits = *reinterpret_cast<const uint4*>(x + i);
#pragma unroll
    for (int e = 0; e < 8; ++e) u.v[e] = rounded(__fmul_rn(as_float(u.v[e]), s));
    *reinterpret_cast<uint4*>(x + i) = u.bits;
  } else {
    for (size_t j = i; j < n && j < i + (VECTOR ? 8 : 1); ++j) x[j] = rounded(__fmul_rn(as_float(x[j]), s));
  }
}

__global__ void rsqrt_kernel(const float* in, float* out, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = rsqrtf(in[i]);
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

gw_status check_norm_shape(uint32_t rows, uint32_t width) {
  if (rows == 0 || width == 0 || width % 8 || width > 16384)
    return fail(GW_INVALID_ARGUMENT, "RMS norm requires rows > 0 and a width divisible by 8, at most 16384");
  return GW_OK;
}

NormArgs norm_args(const void* input, uint32_t rows, uint32_t width) {
  return NormArgs{static_cast<const bf16*>(input), width, reduction_lanes(rows, width), 1.F / float(width)};
}

size_t norm_shared_bytes(uint32_t width, uint32_t lanes, int staged_rows) {
  return size_t(staged_rows) * (width * sizeof(bf16) + lanes * sizeof(float));
}

// A thread for every eight values of a row up to 512, then two or four vectors a thread.
uint32_t norm_vectors(uint32_t width) {
  const uint32_t per_thread = (width / 8 + kNormThreads - 1) / kNormThreads;
  return per_thread <= 2 ? per_thread : 4;
}
uint32_t norm_threads(uint32_t width) {
  const uint32_t nv = norm_vectors(width);
  return ((width / 8 + nv - 1) / nv + 31) / 32 * 32;
}

struct DeviceBuffer {
  void* data = nullptr;
  size_t bytes = 0;
  cudaError_t allocate(size_t n) {
    bytes = n;
    return n ? cudaMalloc(&data, n) : cudaSuccess;
  }
  ~DeviceBuffer() { if (data) cudaFree(data); }
};

constexpr uint32_t kHidden = 2816, kSharedMlp = 2112, kExperts = 128;   // model.h:12-13

}  // namespace

struct gw_ffn_block {
  uint32_t capacity = 0, rows = 0;
  int policy = GW_POLICY_ALWAYS, phase = GW_PHASE_PREFILL;
  cudaStream_t stream = nullptr;
  gw_projection_workspace* projections = nullptr;
  gw_moe_workspace* moe = nullptr;
  // The shared MLP runs on a stream of its own beside the router, the routing and the experts' input, which leave most of
  // the GPU idle at small row counts, and fills the tails of the experts' GEMMs at large ones (one stream -> two, us: NVFP4
  // 8 rows 100.7 -> 95.1, 470 rows 231.8 -> 213.1, 4000 rows 472.8 -> 445.5; BF16 8 rows 172 -> 149).  So the router has a
  // plan apart from the shared MLP's, beyond the rows of router_logits_kernel; such a plan needs no scratch.
  cudaStream_t side = nullptr;
  cudaEvent_t forked = nullptr, joined = nullptr;
  gw_bf16_plan* router_plan = nullptr;
  DeviceBuffer buffers;                  // one allocation, carved below
  bf16 *normalized = nullptr, *router_input = nullptr, *expert_input = nullptr, *gate = nullptr, *up = nullptr,
       *product = nullptr, *shared_mlp = nullptr, *logits = nullptr, *routed = nullptr;
  ~gw_ffn_block() {
    if (projections) gw_projection_workspace_destroy(projections);
    if (moe) gw_moe_destroy(moe);
    if (router_plan) gw_bf16_plan_destroy(router_plan);
    if (forked) cudaEventDestroy(forked);
    if (joined) cudaEventDestroy(joined);
    if (side) cudaStreamDestroy(side);
  }
};

extern "C" {

gw_status gw_rms_norm_bf16(const void* input_bf16, const void* weight_bf16, void* output_bf16, uint32_t rows,
                           uint32_t width, void* stream) {
  clear_error();
  if (rows == 0) return GW_OK;
  if (gw_status s = check_norm_shape(rows, width); s != GW_OK) return s;
  if (!input_bf16 || !output_bf16 || !aligned16(input_bf16))
    return fail(GW_INVALID_ARGUMENT, "RMS norm requires a 16-byte aligned input and an output");
  const NormArgs a = norm_args(input_bf16, rows, width);
  const uint32_t nv = norm_vectors(width);
  GW_CUDA_CHECK(launch_pdl_shared(nv == 1 ? rms_norm_kernel<1> : nv == 2 ? rms_norm_kernel<2> : rms_norm_kernel<4>, rows, norm_threads(width),
                                  norm_shared_bytes(width, a.lanes, 1), as_stream(stream), a, static_cast<const bf16*>(weight_bf16),
                                  static_cast<bf16*>(output_bf16)),
                "RMS norm");
  return GW_OK;
}

gw_status gw_rms_norm_feedforward_bf16(const void* input_bf16, const void* shared_weight, const void* router_weight,
                                       const void* expert_weight, void* shared_bf16, void* router_bf16,
                                       void* expert_bf16, uint32_t rows, uint32_t width, void* stream) {
  clear_error();
  if (rows == 0) return GW_OK;
  if (gw_status s = check_norm_shape(rows, width); s != GW_OK) return s;
  if (!input_bf16 || !aligned16(input_bf16) || !shared_weight || !router_weight || !expert_weight || !shared_bf16 ||
      !router_bf16 || !expert_bf16)
    return fail(GW_INVALID_ARGUMENT, "feed-forward norm requires its input, three weights and three outputs");
  const NormArgs a = norm_args(input_bf16, rows, width);
  const FeedForwardNormArgs f{static_cast<const bf16*>(shared_weight), static_cast<const bf16*>(router_weight),
                              static_cast<const bf16*>(expert_weight), static_cast<bf16*>(shared_bf16),
                              static_cast<bf16*>(router_bf16), static_cast<bf16*>(expert_bf16),
                              1.F / std::sqrt(float(width))};
  const uint32_t nv = norm_vectors(width);
  GW_CUDA_CHECK(launch_pdl_shared(nv == 1   ? rms_norm_feedforward_kernel<1>
                                  : nv == 2 ? rms_norm_feedforward_kernel<2>
                                            : rms_norm_feedforward_kernel<4>,
                                  rows, norm_threads(width), norm_shared_bytes(width, a.lanes, 1), as_stream(stream), a, f),
                "feed-forward norm");
  return GW_OK;
}

gw_status gw_ffn_tail_bf16(const void* shared_mlp_bf16, const void* routed_bf16, const void* norm_shared_weight,
                           const void* norm_routed_weight, const void* norm_sum_weight, const void* layer_scalar_bf16,
                           void* hidden_bf16, uint32_t rows, uint32_t width, void* stream) {
  clear_error();
  if (rows == 0) return GW_OK;
  if (gw_status s = check_norm_shape(rows, width); s != GW_OK) return s;
  if (!shared_mlp_bf16 || !routed_bf16 || !aligned16(shared_mlp_bf16) || !aligned16(routed_bf16) || !norm_shared_weight ||
      !norm_routed_weight || !norm_sum_weight || !layer_scalar_bf16 || !hidden_bf16)
    return fail(GW_INVALID_ARGUMENT, "feed-forward tail requires two 16-byte aligned inputs, three norm weights, "
                                     "the layer scalar and the hidden state");
  const NormArgs a = norm_args(shared_mlp_bf16, rows, width);
  const TailArgs t{static_cast<const bf16*>(shared_mlp_bf16), static_cast<bf16*>(const_cast<void*>(routed_bf16)),
                   static_cast<const bf16*>(norm_shared_weight), static_cast<const bf16*>(norm_routed_weight),
                   static_cast<const bf16*>(norm_sum_weight), static_cast<const bf16*>(layer_scalar_bf16),
                   static_cast<bf16*>(hidden_bf16), nullptr, nullptr, nullptr};
  const size_t shared_bytes = norm_shared_bytes(width, a.lanes, 2);
  const uint32_t nv = norm_vectors(width);
  const auto kernel = nv == 1 ? ffn_tail_kernel<1, false> : nv == 2 ? ffn_tail_kernel<2, false> : ffn_tail_kernel<4, false>;
  static bool raised[kMaxDeviceSlots] = {};
  if (shared_bytes > 48 * 1024 && !raised[current_device_slot()]) {   // only rows of more than 12000 values: four vectors a thread
    GW_CUDA_CHECK(cudaFuncSetAttribute(ffn_tail_kernel<4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 80 * 1024),
                  "feed-forward tail shared memory");
    raised[current_device_slot()] = true;
  }
  GW_CUDA_CHECK(launch_pdl_shared(kernel, rows, norm_threads(width), shared_bytes, as_stream(stream), a, t), "feed-forward tail");
  return GW_OK;
}

gw_status gw_add_bf16(const void* a_bf16, const void* b_bf16, void* output_bf16, uint64_t count, void* stream) {
  clear_error();
  if (count == 0) return GW_OK;
  if (!a_bf16 || !b_bf16 || !output_bf16) return fail(GW_INVALID_ARGUMENT, "add requires three buffers");
  const bool vector = aligned16(a_bf16) && aligned16(b_bf16) && aligned16(output_bf16);
  const uint64_t per_block = vector ? 2048 : 256;
  GW_CUDA_CHECK(launch_pdl(vector ? add_kernel<true> : add_kernel<false>, unsigned((count + per_block - 1) / per_block), 256, as_stream(stream),
                           static_cast<const bf16*>(a_bf16), static_cast<const bf16*>(b_bf16), static_cast<bf16*>(output_bf16), size_t(count)),
                "add");
  return GW_OK;
}

gw_status gw_scale_bf16(void* values_bf16, const void* scalar_bf16, uint64_t count, void* stream) {
  clear_error();
  if (count == 0) return GW_OK;
  if (!values_bf16 || !scalar_bf16) return fail(GW_INVALID_ARGUMENT, "scale requires values and a device scalar");
  const bool vector = aligned16(values_bf16);
  const uint64_t per_block = vector ? 2048 : 256;
  GW_CUDA_CHECK(launch_pdl(vector ? scale_kernel<true> : scale_kernel<false>, unsigned((count + per_block - 1) / per_block), 256, as_stream(stream),
                           static_cast<bf16*>(values_bf16), static_cast<const bf16*>(scalar_bf16), size_t(count)),
                "scale");
  return GW_OK;
}

gw_status gw_debug_rsqrt(const float* host_in, float* host_out, uint32_t count) {
  clear_error();
  if (count == 0) return GW_OK;
  if (!host_in || !host_out) return fail(GW_INVALID_ARGUMENT, "rsqrt probe requires two host arrays");
  DeviceBuffer in, out;
  GW_CUDA_CHECK(in.allocate(size_t(count) * 4), "rsqrt probe");
  GW_CUDA_CHECK(out.allocate(size_t(count) * 4), "rsqrt probe");
  GW_CUDA_CHECK(cudaMemcpy(in.data, host_in, size_t(count) * 4, cudaMemcpyHostToDevice), "rsqrt probe");
  rsqrt_kernel<<<(count + 255) / 256, 256>>>(static_cast<const float*>(in.data), static_cast<float*>(out.data), count);
  GW_CUDA_CHECK(cudaGetLastError(), "rsqrt probe");
  GW_CUDA_CHECK(cudaMemcpy(host_out, out.data, size_t(count) * 4, cudaMemcpyDeviceToHost), "rsqrt probe");
  return GW_OK;
}

uint32_t gw_rms_norm_reduction_lanes(uint32_t rows, uint32_t width) { return reduction_lanes(rows, width); }

// ---------------------------------------------------------------------------------------------------

gw_status gw_ffn_block_create(const gw_ffn_block_weights* layers, uint32_t count, uint32_t max_rows, int policy,
                              uint32_t moe_flags, void* stream, gw_ffn_block** block) {
  clear_error();
  if (!block || !layers || count == 0 || max_rows == 0 || max_rows > 65536)
    return fail(GW_INVALID_ARGUMENT, "feed-forward block requires layers and 1..65536 rows");
  std::vector<gw_projection> bindings;
  for (uint32_t l = 0; l < count; ++l) {
    const gw_ffn_block_weights& w = layers[l];
    if (w.gate.input != kHidden || w.gate.output != kSharedMlp || w.up.input != kHidden || w.up.output != kSharedMlp ||
        w.down.input != kSharedMlp || w.down.output != kHidden)
      return fail(GW_INVALID_ARGUMENT, "shared MLP projections must be 2816 -> 2112 -> 2816");
    if (!w.router_proj) return fail(GW_INVALID_ARGUMENT, "router projection is required");
    bindings.push_back(w.gate);
    bindings.push_back(w.up);
    bindings.push_back(w.down);
  }
  auto b = std::unique_ptr<gw_ffn_block>(new (std::nothrow) gw_ffn_block());
  if (!b) return fail(GW_CUDA_ERROR, "out of host memory");
  b->capacity = max_rows;
  b->policy = policy;
  b->stream = as_stream(stream);
  gw_status status = gw_projection_workspace_create(bindings.data(), uint32_t(bindings.size()), max_rows, policy, stream,
                                                    &b->projections);
  if (status != GW_OK) return status;
  status = gw_moe_create_ex(max_rows, moe_flags, &b->moe);
  if (status != GW_OK) return status;
  const size_t wide = align_up(size_t(max_rows) * kHidden * sizeof(bf16), 256);
  const size_t narrow = align_up(size_t(max_rows) * kSharedMlp * sizeof(bf16), 256);
  const size_t scores = align_up(size_t(max_rows) * kExperts * sizeof(bf16), 256);
  GW_CUDA_CHECK(b->buffers.allocate(5 * wide + 3 * narrow + scores), "feed-forward block buffers");
  GW_CUDA_CHECK(cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking), "feed-forward block stream");
  GW_CUDA_CHECK(cudaEventCreateWithFlags(&b->forked, cudaEventDisableTiming), "feed-forward block event");
  GW_CUDA_CHECK(cudaEventCreateWithFlags(&b->joined, cudaEventDisableTiming), "feed-forward block event");
  auto* cursor = static_cast<unsigned char*>(b->buffers.data);
  auto carve = [&cursor](size_t bytes) {
    bf16* p = reinterpret_cast<bf16*>(cursor);
    cursor += bytes;
    return p;
  };
  b->normalized = carve(wide);
  b->router_input = carve(wide);
  b->expert_input = carve(wide);
  b->shared_mlp = carve(wide);
  b->routed = carve(wide);
  b->gate = carve(narrow);
  b->up = carve(narrow);
  b->product = carve(narrow);
  b->logits = carve(scores);
  *block = b.release();
  return GW_OK;
}

void gw_ffn_block_destroy(gw_ffn_block* block) { delete block; }

size_t gw_ffn_block_bytes(const gw_ffn_block* b) {
  return b ? b->buffers.bytes + gw_projection_workspace_bytes(b->projections) + gw_moe_bytes(b->moe) : 0;
}

gw_status gw_ffn_block_prepare(gw_ffn_block* b, uint32_t rows, int phase) {
  clear_error();
  if (!b || rows == 0 || rows > b->capacity) return fail(GW_INVALID_ARGUMENT, "feed-forward block: invalid rows");
  // The router's plan first, beside the present one: what follows either prepares the projections too or leaves all as it was.
  gw_bf16_plan* plan = nullptr;
  if (b->rows != rows && rows > kRouterRows)
    if (const gw_status created = gw_bf16_plan_create(rows, kHidden, kExperts, &plan); created != GW_OK) return created;
  const gw_status status = gw_projection_workspace_prepare(b->projections, rows, phase);
  if (status != GW_OK) {
    if (plan) gw_bf16_plan_destroy(plan);
    return status;
  }
  if (b->rows != rows) {
    if (b->router_plan) gw_bf16_plan_destroy(b->router_plan);
    b->router_plan = plan;
  }
  b->rows = rows;
  b->phase = phase;
  return GW_OK;
}

gw_status gw_ffn_block_run(gw_ffn_block* b, const gw_ffn_block_weights* weights, void* hidden_bf16) {
  clear_error();
  if (!b || !weights || !hidden_bf16 || b->rows == 0)
    return fail(GW_INVALID_ARGUMENT, "prepare the feed-forward block before run");
  const gw_ffn_block_weights& w = *weights;
  if (!w.pre_feedforward_norm || !w.router_scale || !w.pre_feedforward_norm_2 || !w.post_feedforward_norm_1 ||
      !w.post_feedforward_norm_2 || !w.post_feedforward_norm || !w.layer_scalar || !w.router_proj ||
      !w.router_per_expert_scale || !w.experts)
    return fail(GW_INVALID_ARGUMENT, "feed-forward block: a weight is missing");
  if (!aligned16(w.router_proj)) return fail(GW_INVALID_ARGUMENT, "feed-forward block requires a 16-byte aligned router projection");
  const uint32_t rows = b->rows;
  void* s = b->stream;
  gw_status status = gw_rms_norm_feedforward_bf16(hidden_bf16, w.pre_feedforward_norm, w.router_scale,
                                                  w.pre_feedforward_norm_2, b->normalized, b->router_input,
                                                  b->expert_input, rows, kHidden, s);
  if (status != GW_OK) return status;
  // shared MLP (batched_executor.cu:256-259)
  GW_CUDA_CHECK(cudaEventRecord(b->forked, as_stream(s)), "feed-forward block fork");
  GW_CUDA_CHECK(cudaStreamWaitEvent(b->side, b->forked, 0), "feed-forward block fork");
  // in front of every launch of both streams is one of this call's own, which writes no weights
  const auto shared_mlp = [&]() {
    bool product_done = false;
    gw_status st = projection_workspace_run_geglu(b->projections, w.gate, w.up, b->normalized, b->product, b->side, true,
                                                  &product_done);
    if (st == GW_OK && !product_done) {
      bool done = false;
      st = projection_workspace_run_mlp(b->projections, w.gate, w.up, w.down, b->normalized, b->product, b->shared_mlp, b->side, &done);
      if (st != GW_OK || done) return st;
      st = projection_workspace_run_on(b->projections, &w.gate, b->normalized, b->gate, b->side, true);
      if (st == GW_OK) st = projection_workspace_run_on(b->projections, &w.up, b->normalized, b->up, b->side, true);
      if (st == GW_OK) st = gw_gelu_tanh_multiply_bf16(b->gate, b->up, b->product, uint64_t(rows) * kSharedMlp, b->side);
    }
    return st == GW_OK ? projection_workspace_run_on(b->projections, &w.down, b->product, b->shared_mlp, b->side, true) : st;
  };
  status = shared_mlp();
  // a failed call still brings its side stream back
  const cudaError_t recorded = cudaEventRecord(b->joined, b->side);
  if (status != GW_OK) {
    (void)cudaStreamWaitEvent(as_stream(s), b->joined, 0);
    return status;
  }
  GW_CUDA_CHECK(recorded, "feed-forward block join");
  // router logits and the experts (batched_executor.cu:262-266)
  if (rows <= kRouterRows) {
    const cudaError_t launched =
        launch_pdl(router_logits_kernel, dim3(kRouterExperts / 16, (rows + 7) / 8), kRouterThreads, as_stream(s),
                   reinterpret_cast<const uint4*>(b->router_input), static_cast<const uint4*>(w.router_proj), b->logits, rows);
    if (launched != cudaSuccess) status = fail(GW_CUDA_ERROR, std::string("router logits: ") + cudaGetErrorString(launched));
  } else {
    status = run_bf16_plan(b->router_plan, b->router_input, w.router_proj, b->logits, nullptr, 0, as_stream(s), true);
  }
  MoeCombineInput combine;
  if (status == GW_OK)
    status = moe_run_to_down(b->moe, b->expert_input, b->logits, w.router_per_expert_scale, w.experts, rows, w.has_bf16, w.has_fp8,
                             w.has_nvfp4, gw_nvfp4_fp4_activations(b->policy, b->phase), as_stream(s), &combine);
  GW_CUDA_CHECK(cudaStreamWaitEvent(as_stream(s), b->joined, 0), "feed-forward block join");
  if (status != GW_OK) return status;
  // the experts' weighted sum and the block's tail in one launch
  const NormArgs a = norm_args(b->shared_mlp, rows, kHidden);
  const TailArgs t{b->shared_mlp, b->routed, static_cast<const bf16*>(w.post_feedforward_norm_1),
                   static_cast<const bf16*>(w.post_feedforward_norm_2), static_cast<const bf16*>(w.post_feedforward_norm),
                   static_cast<const bf16*>(w.layer_scalar), static_cast<bf16*>(hidden_bf16), static_cast<const uint4*>(combine.down),
                   combine.inverse, combine.weights};
  static_assert(kHidden / 8 == kBlockThreads, "one vector a thread");
  GW_CUDA_CHECK(launch_pdl_shared(ffn_tail_kernel<1, true>, rows, norm_threads(kHidden), norm_shared_bytes(kHidden, a.lanes, 2), as_stream(s), a, t),
                "feed-forward tail");
  moe_mark_combined(b->moe, as_stream(s));
  return GW_OK;
}

const void* gw_ffn_block_buffer(const gw_ffn_block* b, int which) {
  if (!b) return nullptr;
  switch (which) {
    case GW_FFN_NORMALIZED: return b->normalized;
    case GW_FFN_ROUTER_INPUT: return b->router_input;
    case GW_FFN_EXPERT_INPUT: return b->expert_input;
    case GW_FFN_SHARED_MLP: return b->shared_mlp;
    case GW_FFN_ROUTER_LOGITS: return b->logits;
    case GW_FFN_ROUTED: return b->routed;
    default: return nullptr;
  }
}

gw_moe_workspace* gw_ffn_block_moe(gw_ffn_block* b) { return b ? b->moe : nullptr; }

}  // extern "C"
