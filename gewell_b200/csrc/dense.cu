#include "dense.h"
#include "gemm_pair.h"
#include "gemm_pair_wide.h"

#include <algorithm>
#include <cstdlib>
#include <string>

namespace gw {

DenseTuning DenseTuning::from_environment() {
  DenseTuning tuning;
  if (const char* forced = std::getenv("GW_DENSE_FORM")) tuning.form = forced[0];
  if (const char* forced = std::getenv("GW_DENSE_BLOCK_N")) tuning.block_n = std::atoi(forced);
  tuning.no_pair = std::getenv("GW_DENSE_NO_PAIR") != nullptr;
  tuning.no_split = std::getenv("GW_DENSE_NO_SPLIT") != nullptr;
  return tuning;
}

bool dense_uses_swap_form(const DenseTuning& tuning, uint32_t rows) {
  if (tuning.form == 's' && rows <= 128) return true;
  if (tuning.form == 'd') return false;
  return rows <= 128;
}

int dense_block_n(const DenseTuning& tuning, uint32_t rows) {
  if (dense_uses_swap_form(tuning, rows)) return rows <= 32 ? 32 : rows <= 64 ? 64 : 128;
  if (tuning.block_n == 128 || tuning.block_n == 256) return tuning.block_n;
  return 256;
}

namespace {
size_t split_counter_bytes(const DenseTuning& tuning, uint32_t rows, uint32_t n) {
  const int block_n = dense_block_n(tuning, rows);
  const size_t tiles = size_t((n + 127) / 128) * ((rows + block_n - 1) / block_n);
  return align_up(tiles * sizeof(int32_t), 256);
}
}  // namespace

// Where the weight-streaming kernel is the faster one for rows <= 16 (B200, both timed back to back, us; old = activation
// quantiser + tcgen05 swap form): NVFP4 16x2816x2816 15.3 -> 9.3, 8x5376x43008 32.6 -> 33, 1x21504x5376 24.1 -> 20.9; FP8
// 8x5376x43008 46.3 -> 42.6.  It saves the quantiser's launch and the tensor-memory prologue; what it pays is that every SM
// reads and quantises all of the activations: about 1 us per 16K values, which meets the gain at 64K.  Nine and more
// rows need a second token group (half as many instructions again per weight byte), which only small matrices hide.
// W4A16 has no other kernel that reads the packed weights.
bool stream_pays(StreamKind kind, const StreamPlan& plan, uint32_t rows, uint32_t k, size_t n) {
  if (!plan.usable || kind == StreamKind::w4a16) return plan.usable;
  const size_t values = size_t(rows) * k;
  const size_t bytes = n * k * (kind == StreamKind::w4a4 ? 9 : kind == StreamKind::w8a8 ? 16 : 32) / 16;
  if (values > 65536) return false;
  if (plan.tiles == 2 && values > 46 * 1024 && bytes > (size_t(20) << 20)) return false;
  // BF16 tokens of more than 8192 values need several slabs: twice the sums
  return kind != StreamKind::w16a16 || plan.slabs == 1 || bytes <= (size_t(48) << 20);
}

size_t dense_split_bytes(const DenseTuning& tuning, uint32_t rows, uint32_t n) {
  (void)n;
  if (!dense_uses_swap_form(tuning, rows) || tuning.no_split) return 0;
  return size_t(2) * sm_count() * 128 * dense_block_n(tuning, rows) * sizeof(float);
}

size_t DenseDescriptors::split_bytes(uint32_t rows, uint32_t n) const {
  if (split_counters == nullptr) return 0;
  return align_up(std::max(dense_split_bytes(tuning, rows, n), stream.usable ? stream.workspace_bytes : 0), 256);
}

cudaError_t DenseDescriptors::allocate_split_counters(GemmKind kind, uint32_t rows, uint32_t k, uint32_t n) {
  if (dense_split_bytes(tuning, rows, n) == 0) return cudaSuccess;
  size_t bytes = split_counter_bytes(tuning, rows, n);
  if (tuning.streams()) {
    const StreamKind as = kind == GemmKind::nvfp4 ? StreamKind::w4a4 : kind == GemmKind::fp8 ? StreamKind::w8a8 : StreamKind::w16a16;
    stream = plan_stream(as, rows, k, n, false, sm_count());
    stream.usable = stream_pays(as, stream, rows, k, n);
    if (stream.usable) bytes = std::max(bytes, align_up(stream.counter_count * sizeof(int32_t), 256));
  }
  cudaError_t status = cudaMalloc(&split_counters, bytes);
  if (status == cudaSuccess) status = cudaMemset(split_counters, 0, bytes);
  return status;
}

DenseDescriptors::~DenseDescriptors() {
  if (split_counters != nullptr) cudaFree(split_counters);
}

gw_status launch_dense_stream(const StreamProblem& q, DenseDescriptors* cache, cudaStream_t stream, bool* done) {
  *done = cache->stream.usable && stream_aligned(q);
  if (!*done) return GW_OK;
  std::string error;
  if (!cache->stream_maps.get(q.kind, q.first, cache->stream.physical_n, q.k, &error))
    return fail(GW_CUDA_ERROR, "weight descriptor: " + error);
  GW_CUDA_CHECK(launch_stream(q, cache->stream, cache->stream_maps, cache->stream_maps, stream), "weight-streaming projection");
  return GW_OK;
}

namespace {

// FP8 and BF16 with more rows than the swap form takes: channels on the lanes of a CTA pair.
gw_status launch_dense_pair_wide(const DenseProblem& q, uint64_t row_bytes, DenseDescriptors* cache, cudaStream_t stream) {
  std::string error;
  if (cache->token_tile == 0) cache->token_tile = pair_wide_tile_rows(q.rows, q.n, sm_count());
  if (cache->weight_half != q.weight) {
    if (!encode_tensor_map_2d(&cache->weight_half_map, q.weight, row_bytes, q.n, 128, &error))
      return fail(GW_CUDA_ERROR, "weight descriptor: " + error);
    cache->weight_half = q.weight;
  }
  if (cache->activations != q.activations) {
    if (!encode_tensor_map_2d(&cache->activation_map, q.activations, row_bytes, q.rows, uint32_t(cache->token_tile / 2), &error))
      return fail(GW_CUDA_ERROR, "activation descriptor: " + error);
    cache->activations = q.activations;
  }
  PairWideParams pair{};
  pair.map_weights = cache->weight_half_map;
  pair.map_tokens = cache->activation_map;
  pair.k_stages = int32_t((row_bytes + 127) / 128);
  pair.last_kb = int32_t((row_bytes - uint64_t(pair.k_stages - 1) * 128 + 31) / 32);
  pair.rows = int32_t(q.rows);
  pair.n = int32_t(q.n);
  pair.channel_tiles = int32_t((q.n + 255) / 256);
  pair.token_tiles = int32_t((q.rows + cache->token_tile - 1) / cache->token_tile);
  pair.tile_rows = cache->token_tile;
  pair.out = q.output;
  pair.ld_out = q.n;
  pair.alpha = q.alpha;
  pair.channel_alpha = q.channel_alpha;
  pair.error = q.error;
  GW_CUDA_CHECK(launch_gemm_pair_wide(q.kind == GemmKind::fp8, pair, sm_count(), stream),
                q.kind == GemmKind::fp8 ? "FP8 CTA-pair tensor-core GEMM" : "BF16 CTA-pair tensor-core GEMM");
  return GW_OK;
}

}  // namespace

gw_status launch_dense(const DenseProblem& q, DenseDescriptors* cache, cudaStream_t stream) {
  const DenseTuning& tuning = cache->tuning;
  const bool swap = dense_uses_swap_form(tuning, q.rows);
  const int block_n = dense_block_n(tuning, q.rows);
  const bool fp4 = q.kind == GemmKind::nvfp4;
  const uint64_t row_bytes = fp4 ? q.k / 2 : (q.kind == GemmKind::bf16 ? uint64_t(2) * q.k : q.k);
  std::string error;
  // Outputs of these kinds are 16-byte aligned and a multiple of 8 wide (plan creation and the run check it).
  if (!fp4 && !swap && tuning.form == 0 && tuning.block_n == 0 && !tuning.no_pair)
    return launch_dense_pair_wide(q, row_bytes, cache, stream);
  const bool single_box = !swap && block_n == 256;   // both column halves come from the one weight matrix
  if (cache->weight != q.weight) {
    if (!encode_tensor_map_2d(&cache->weight_map, q.weight, row_bytes, q.n, single_box ? 256 : 128, &error))
      return fail(GW_CUDA_ERROR, "weight descriptor: " + error);
    cache->weight = q.weight;
  }
  if (single_box && fp4 && cache->weight_scales != q.weight_scales) {
    if (!encode_tensor_map_scales(&cache->weight_scale_map, q.weight_scales, q.k / 64, (q.n + 127) / 128, 2, &error))
      return fail(GW_CUDA_ERROR, "weight scale descriptor: " + error);
    cache->weight_scales = q.weight_scales;
  }
  if (cache->activations != q.activations) {
    if (!encode_tensor_map_2d(&cache->activation_map, q.activations, row_bytes, q.rows, swap ? block_n : 128, &error))
      return fail(GW_CUDA_ERROR, "activation descriptor: " + error);
    cache->activations = q.activations;
  }
  // NVFP4 prefill: the CTA-pair kernel (each CTA stages half of the weight tile) unless disabled
  if (fp4 && single_box && q.rows >= 256 && !tuning.no_pair) {
    if (cache->weight_half != q.weight) {
      if (!encode_tensor_map_2d(&cache->weight_half_map, q.weight, row_bytes, q.n, 128, &error))
        return fail(GW_CUDA_ERROR, "weight descriptor: " + error);
      cache->weight_half = q.weight;
    }
    PairGemmParams pair{};
    pair.map_tokens = cache->activation_map;
    pair.map_weights = cache->weight_half_map;
    pair.map_weight_scales = cache->weight_scale_map;
    pair.sf_tokens = q.activation_scales;
    pair.token_row_blocks = int32_t((q.rows + 127) / 128);
    pair.k = int32_t(q.k);
    pair.rows = int32_t(q.rows);
    pair.n = int32_t(q.n);
    pair.l_tiles = int32_t((q.rows + 255) / 256);
    pair.c_tiles = int32_t((q.n + 255) / 256);
    pair.out = q.output;
    pair.ld_out = q.n;
    pair.alpha = q.alpha;
    pair.error = q.error;
    GW_CUDA_CHECK(launch_gemm_pair(pair, sm_count(), stream), "NVFP4 CTA-pair tensor-core GEMM");
    return GW_OK;
  }
  GemmParams params{};
  GemmGroup& g = params.single;
  params.groups = nullptr;
  params.num_groups = 1;
  params.k = int32_t(q.k);
  params.out = q.output;
  params.ld_out = q.n;
  params.error = q.error;
  g.alpha[0] = g.alpha[1] = q.alpha;
  g.channel_alpha = q.channel_alpha;
  g.map_l = -1;
  g.map_c[0] = g.map_c[1] = -1;
  if (swap) {
    params.early_weights = 1;   // weights are never written by the activation-quantise kernel before this launch
    params.map_l = cache->weight_map;
    params.map_c = cache->activation_map;
    params.c_rows_per_tile = block_n;
    g.sf_l = q.weight_scales;
    g.l_rows = int32_t(q.n);
    g.l_tiles = int32_t((q.n + 127) / 128);
    g.sf_c[0] = g.sf_c[1] = q.activation_scales;
    g.c_rows = int32_t(q.rows);
    g.c_tiles = int32_t((q.rows + block_n - 1) / block_n);
    g.c_half_stride = 0;
  } else {
    params.map_l = cache->activation_map;
    params.map_c = cache->weight_map;
    params.c_rows_per_tile = block_n;
    g.sf_l = q.activation_scales;
    g.l_rows = int32_t(q.rows);
    g.l_tiles = int32_t((q.rows + 127) / 128);
    g.sf_c[0] = g.sf_c[1] = q.weight_scales;
    g.c_rows = int32_t(q.n);
    g.c_tiles = int32_t((q.n + block_n - 1) / block_n);
    g.c_half_stride = block_n > 128 ? 128 : 0;
    if (single_box) {
      params.c_single_box = 1;
      if (fp4) params.map_sfc = cache->weight_scale_map;
    }
  }
  params.total_work = g.l_tiles * g.c_tiles;
  int grid = params.total_work < sm_count() ? params.total_work : sm_count();
  if (swap && q.split_workspace != nullptr && cache->split_counters != nullptr) {
    params.split_counters = cache->split_counters;
    params.split_partials = static_cast<float*>(q.split_workspace);
    const long long stages = (long long)gemm_tc_k_stages(q.kind, GemmEpilogue::swap_store, row_bytes) * params.total_work;
    grid = stages < sm_count() ? int(stages) : sm_count();
  }
  GW_CUDA_CHECK(launch_gemm_tc(q.kind, swap ? GemmEpilogue::swap_store : GemmEpilogue::direct_store, block_n, params,
                               grid, stream),
                fp4 ? "NVFP4 tensor-core GEMM" : (q.kind == GemmKind::bf16 ? "BF16 tensor-core GEMM" : "FP8 tensor-core GEMM"));
  return GW_OK;
}

}  // namespace gw
