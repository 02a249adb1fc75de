#include "dense.h"
#include "gemm_pair.h"
#include "gemm_pair_wide.h"

#include <algorithm>
#include <cmath>
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

namespace {
int swap_block_n(uint32_t rows) { return rows <= 32 ? 32 : rows <= 64 ? 64 : 128; }
}  // namespace

int dense_block_n(const DenseTuning& tuning, uint32_t rows) {
  if (dense_uses_swap_form(tuning, rows)) return swap_block_n(rows);
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

// Where the weight-streaming kernel is the faster one.  It saves the quantiser's launch and the tensor-memory prologue; what it
// pays is that every SM reads and quantises all of the activations, that some SMs have one row block more than others, and, with
// several slabs (!StreamPlan::whole), 2 us for adding sums in a second pass.  Measured against activation quantiser + tcgen05 swap form
// (B200, rotating weights, passes of a CUDA graph; time of the streaming kernel over the other's):
//   whole row blocks    FP8, 1 to 8 rows, K 1024 .. 8192, N 512 .. 43008, rows * K up to 44 K    0.58 .. 1.02, 8x5376x16384 1.06,
//                                                                                8 rows, K up to 2048, N 6144 .. 9600 1.02 .. 1.06
//                       BF16 the same                                                            0.55 .. 1.01, 8x5376x16384 1.05
//                       NVFP4, N up to 4736 (one block an SM), rows * K up to 24 K   0.67 .. 1.04; more 0.97 .. 1.09
//                              N up to 9472, rows * K up to 6 K      0.89 .. 0.98, K 512 1.02 .. 1.08; more 0.98 .. 1.21
//                              N up to 18944 (one wave of the swap form's tiles)  0.94 .. 1.22
//                              beyond, rows * K up to 24 K           0.68 .. 1.00; 8x5376x43008 1.04
//   several slabs       NVFP4 and FP8 up to N 512 0.84 .. 0.97, beyond 0.82 .. 1.41; BF16 up to N 2048 0.78 .. 1.16, beyond 0.88 .. 1.65
// In us: NVFP4 1x2816x2816 5.3 / 6.9, 1x5376x21504 15.2 / 18.2, 8x2816x8192 8.3 / 7.6; FP8 1x5376x5376 6.7 / 11.5 (K 4096), 4x5376x43008 36.4 /
// 40.6; BF16 8x2816x4096 7.3 / 9.2.  W4A16 has no other kernel that reads the packed weights.
bool stream_pays(StreamKind kind, const StreamPlan& plan, uint32_t rows, uint32_t k, size_t n) {
  if (!plan.usable || kind == StreamKind::w4a16) return plan.usable;
  const size_t values = size_t(rows) * k, sms = size_t(sm_count());
  if (!plan.whole) return k <= 16384 && values <= 24 * 1024 && n <= (kind == StreamKind::w16a16 ? 2048 : 512);
  if (kind != StreamKind::w4a4) return values <= 44 * 1024;
  if (n <= 32 * sms || n > 128 * sms) return values <= 24 * 1024;
  return n <= 64 * sms && values <= 6 * 1024;
}

namespace {
// With GeGLU in front of the quantiser every SM computes all of it.  Over GeGLU + quantiser + swap form (passes of a graph |
// launched one by one): one slab and at most 12 K values 0.80 .. 1.44 | 0.66 .. 1.16; more values 0.88 .. 1.86 | 0.82 .. 1.46, several
// slabs 0.90 .. 1.80 | 0.91 .. 1.72.
bool stream_gelu_pays(const StreamPlan& plan, uint32_t rows, uint32_t k) { return plan.whole && size_t(rows) * k <= 12 * 1024; }
}  // namespace

// Rows up to which W4A16 runs as launches of the weight-streaming kernel, sixteen rows each, instead of dequantising the
// weights for a BF16 GEMM.  The streamed product does not round the weights to BF16, the dequantised one does, as the reference
// does it: the line changes results within that rounding.  (MLP of hidden -> n -> hidden, us, streamed / dequantised):
//   5376 -> 21504     16 rows 100 / 285    32 rows 200 / 287    48 rows 300 / 291
//   4096 -> 11008              57 / 126             113 / 126             169 / 130
//   2816 -> 8192               48 / 83               93 / 84              137 / 87
//   2816 -> 2176               23 / 48               45 / 49               68 / 54
//   1408 -> 4096               27 / 47               54 / 48               80 / 50
constexpr uint32_t kW4a16Rows = 32;

// Gate, up and GeGLU as one streaming launch (n: channels of each).  Where the two matrices lie apart it stands against two
// projections and a GeGLU kernel, where they are joined against one GEMM whose GeGLU rides in the next quantiser (BF16: a kernel
// of its own).  Whole chains of hidden -> n -> hidden with joined matrices, hidden 1152 .. 5376, 1 to 8 rows, time over the other way
// (passes of a graph):
//   n up to 4224, rows * K up to 24 K   NVFP4 0.98 .. 1.11, FP8 0.96 .. 1.13, BF16 0.90 .. 1.14; apart 0.64 .. 1.04 (launched one by one)
//   BF16 beyond                         0.89 .. 0.99
//   FP8, matrices of 64 MB and more     0.92 .. 1.00; less: one row 0.92 .. 0.98, more 0.97 .. 1.27
//   NVFP4, 48 MB and more, rows * K up to 22 K   0.86 .. 0.99, more 1.00 .. 1.02; less: one row 0.92 .. 1.05, more 0.99 .. 1.25
// In us: NVFP4 1x5376x21504 47.9 / 51.5, 1x4096x11008 24.6 / 28.7; FP8 1x5376x21504 63.5 / 65.9; BF16 4x3584x12544 49.4 / 55.6.
bool stream_pair_pays(StreamKind kind, const StreamPlan& plan, uint32_t rows, uint32_t k, size_t n) {
  if (!plan.usable || kind == StreamKind::w4a16) return plan.usable;
  const size_t bytes = 2 * n * k * (kind == StreamKind::w4a4 ? 9 : kind == StreamKind::w8a8 ? 16 : 32) / 16;
  const size_t values = size_t(rows) * k;
  if (n <= 4224) return values <= 24 * 1024;
  if (!plan.whole) return bytes >= (size_t(96) << 20) && values <= 8192;
  if (kind == StreamKind::w16a16 || rows == 1) return true;
  return kind == StreamKind::w8a8 ? bytes >= (size_t(64) << 20) : bytes >= (size_t(48) << 20) && values <= 22 * 1024;
}

namespace {
// CTAs of a swap-form launch that divides the K loops of its `tiles` among them, or 0: whole tiles are faster.
// Dividing costs about 3.4 us (32 token columns; 4.3 with 64, 8 with 128) for the partial sums, the fence, the counter and
// the reading back, and more with more than four CTAs a tile; it gains what an uneven or nearly empty wave of tiles
// leaves idle.  A K stage takes 0.28 (NVFP4) / 0.5 (FP8, two slabs) / 0.2 us (BF16) of latency, and no less than its bytes
// at 5.2 TB/s over the CTAs that run.  Measured, divided over all SMs -> whole tiles (us): NVFP4 32x2816x2816 12.8 -> 7.6,
// 64x2816x2816 16.3 -> 8.9, 24x5376x8192 14.4 -> 10.4, FP8 64x2816x2816 15.3 -> 8.9; BF16 64x2816x128 stays divided, by
// four: 12.4 -> 9.9.  CTAs that begin in one tile and end in another write two partial tiles, so NVFP4 takes as many for
// every tile: 12x21504x5376 (42 tiles, 148 -> 126 CTAs) 19.2 -> 16.9, 64x8192x5376 18.1 -> 14.4, 100x21504x5376 30.8 -> 25.1.  Their
// parts of K are longer, and a sum of products with block scales rounds where the scales differ widely (outputs that are not the
// nearest BF16 with blocks scaled by 2^-6 .. 2^6, 100x21504x5376, 148 / 126 CTAs 1.3e-3 / 1.6e-3; none with N(0, 1)): so each of these
// CTAs has an accumulator for either half of its part.
int swap_split_grid(GemmKind kind, int tiles, int stages, int block_n) {
  const int sms = sm_count();
  const double latency = kind == GemmKind::nvfp4 ? 0.28 : kind == GemmKind::fp8 ? 0.5 : 0.2;
  const double bytes = kind == GemmKind::nvfp4 ? 18e3 : kind == GemmKind::fp8 ? 32e3 : 16e3;
  const auto stage_us = [&](int ctas) { return std::max(latency, bytes * ctas / 5.2e6); };
  const int whole_grid = std::min(tiles, sms);
  const double whole = double((tiles + whole_grid - 1) / whole_grid) * stages * stage_us(whole_grid);
  int grid = int(std::min<long long>({(long long)(tiles) * stages, (long long)(sms), 4ll * tiles}));
  if (kind == GemmKind::nvfp4 && grid > tiles) grid -= grid % tiles;
  const double divided = double(tiles) * stages / grid * stage_us(grid) + (block_n <= 32 ? 3.4 : block_n <= 64 ? 4.3 : 8.0);
  return divided < whole ? grid : 0;
}
}  // namespace

size_t dense_split_bytes(const DenseTuning& tuning, uint32_t rows) {
  if (!dense_uses_swap_form(tuning, rows) || tuning.no_split) return 0;
  return size_t(2) * sm_count() * 128 * dense_block_n(tuning, rows) * sizeof(float);
}

size_t DenseDescriptors::split_bytes(uint32_t rows) const {
  if (split_counters == nullptr) return 0;
  return align_up(std::max(dense_split_bytes(tuning, rows), stream.usable ? stream.workspace_bytes : 0), 256);
}

cudaError_t DenseDescriptors::allocate_split_counters(GemmKind kind, uint32_t rows, uint32_t k, uint32_t n) {
  if (dense_split_bytes(tuning, rows) == 0) return cudaSuccess;
  size_t bytes = split_counter_bytes(tuning, rows, n);
  if (tuning.streams()) {
    const StreamKind as = kind == GemmKind::nvfp4 ? StreamKind::w4a4 : kind == GemmKind::fp8 ? StreamKind::w8a8 : StreamKind::w16a16;
    stream = plan_stream(as, rows, k, n, false, sm_count());
    stream.usable = stream_pays(as, stream, rows, k, n);
    if (stream.usable) bytes = std::max(bytes, align_up(stream.counter_count * sizeof(int32_t), 256));
  }
  cudaError_t status = cudaMalloc(&split_counters, bytes);
  if (status == cudaSuccess) status = zero_now(split_counters, bytes);
  return status;
}

DenseDescriptors::~DenseDescriptors() {
  if (split_counters != nullptr) cudaFree(split_counters);
}

gw_status launch_dense_stream(const StreamProblem& q, DenseDescriptors* cache, cudaStream_t stream, bool* done) {
  *done = cache->stream.usable && stream_aligned(q) && (!q.gelu || stream_gelu_pays(cache->stream, q.rows, q.k));
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
  if (cache->wide.tile_rows == 0) cache->wide = pair_wide_tiles(q.rows, q.n, int((row_bytes + 127) / 128), sm_count());
  if (cache->weight_half != q.weight) {
    if (!encode_tensor_map_2d(&cache->weight_half_map, q.weight, row_bytes, q.n, 128, &error))
      return fail(GW_CUDA_ERROR, "weight descriptor: " + error);
    cache->weight_half = q.weight;
  }
  if (cache->activations != q.activations) {
    if (!encode_tensor_map_2d(&cache->activation_map, q.activations, row_bytes, q.rows, uint32_t(cache->wide.tile_rows / 2), &error) ||
        !encode_tensor_map_2d(&cache->piece_map, q.activations, row_bytes, q.rows, uint32_t(cache->wide.piece_rows / 2), &error))
      return fail(GW_CUDA_ERROR, "activation descriptor: " + error);
    cache->activations = q.activations;
  }
  PairWideParams pair{};
  pair.map_weights = cache->weight_half_map;
  pair.map_tokens = cache->activation_map;
  pair.map_piece = cache->piece_map;
  pair.k_stages = int32_t((row_bytes + 127) / 128);
  pair.last_kb = int32_t((row_bytes - uint64_t(pair.k_stages - 1) * 128 + 31) / 32);
  pair.rows = int32_t(q.rows);
  pair.n = int32_t(q.n);
  pair.tiles = cache->wide;
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

StreamBook::~StreamBook() {
  if (counters != nullptr) cudaFree(counters);
}

StreamBook::Staged::~Staged() {
  if (counters != nullptr) cudaFree(counters);
}

gw_status StreamBook::stage(uint32_t new_rows, const std::vector<std::pair<uint32_t, uint32_t>>& shapes, size_t workspace_bytes,
                            Staged* staged) const {
  staged->rows = new_rows;
  size_t most = 0;
  const bool allowed = DenseTuning::from_environment().streams();
  for (const auto& [k, n] : shapes)
    for (StreamKind kind : {StreamKind::w4a4, StreamKind::w4a16, StreamKind::w8a8, StreamKind::w16a16})
      for (bool pair : {false, true}) {
        // W4A16 beyond one launch's rows: several launches, each of them reads the packed weights once
        const uint32_t tile = kind == StreamKind::w4a16 && new_rows <= kW4a16Rows ? std::min(new_rows, kStreamMaxRows) : new_rows;
        Entry s;
        s.plan = plan_stream(kind, tile, k, n, pair, sm_count());
        s.plan.usable = allowed && (pair ? stream_pair_pays(kind, s.plan, tile, k, n) : stream_pays(kind, s.plan, tile, k, n));
        if (!s.plan.usable || s.plan.workspace_bytes > workspace_bytes) continue;
        most = std::max(most, s.plan.counter_count);
        staged->entries[Key{int(kind), k, n, pair}] = s;
      }
  if (most * sizeof(int32_t) > counter_bytes) {
    cudaError_t status = cudaMalloc(&staged->counters, most * sizeof(int32_t));
    if (status == cudaSuccess) status = zero_now(staged->counters, most * sizeof(int32_t));
    if (status != cudaSuccess)
      return fail(GW_CUDA_ERROR, std::string("counters of the weight-streaming kernel: ") + cudaGetErrorString(status));
    staged->counter_bytes = most * sizeof(int32_t);
  }
  return GW_OK;
}

void StreamBook::publish(Staged* staged) {
  entries.swap(staged->entries);
  rows = staged->rows;
  if (staged->counters != nullptr) {          // the former ones go with `staged`
    std::swap(counters, staged->counters);
    std::swap(counter_bytes, staged->counter_bytes);
  }
}

gw_status StreamBook::run(const gw_projection& first, const gw_projection* second, const void* input, void* output, bool fp4,
                          void* workspace, bool weights_settled, cudaStream_t s, bool* done) {
  *done = false;
  if (second && (second->storage != first.storage || second->input != first.input || second->output != first.output ||
                 second->physical_output != first.physical_output)) return GW_OK;
  const uint32_t physical = first.storage == GW_STORAGE_NVFP4_W4A4 ? first.physical_output : first.output;
  StreamKind kind = StreamKind::w16a16;
  float input_scale = 1.0F;
  if (first.storage == GW_STORAGE_NVFP4_W4A4) {
    kind = fp4 ? StreamKind::w4a4 : StreamKind::w4a16;
    if (fp4) {
      input_scale = first.nvfp4_input_scale;
      if (second && second->nvfp4_input_scale != input_scale) return GW_OK;
    }
  } else if (first.storage == GW_STORAGE_FP8_W8A8) {
    kind = StreamKind::w8a8;
    input_scale = first.fp8_input_scale;
    if (second && second->fp8_input_scale != input_scale) return GW_OK;
  }
  const auto found = entries.find(Key{int(kind), first.input, physical, second != nullptr});
  if (found == entries.end() || !std::isfinite(1.0F / input_scale) || !(input_scale > 0.0F)) return GW_OK;
  Entry& with = found->second;
  StreamProblem q{kind, std::min(rows, kStreamMaxRows), first.input, first.output, input};
  q.inverse_scale = 1.0F / input_scale;
  const gw_projection* projection[2] = {&first, second};
  StreamMatrix* matrix[2] = {&q.first, &q.second};
  std::string error;
  for (int i = 0; i < (second ? 2 : 1); ++i) {
    const gw_projection& p = *projection[i];
    StreamMatrix& m = *matrix[i];
    if (p.storage == GW_STORAGE_NVFP4_W4A4)
      m = StreamMatrix{p.nvfp4_data, p.nvfp4_scales, fp4 ? p.nvfp4_input_scale * p.nvfp4_weight_scale : p.nvfp4_weight_scale, nullptr};
    else if (p.storage == GW_STORAGE_FP8_W8A8)
      m = StreamMatrix{p.fp8_data, nullptr, p.fp8_input_scale * p.fp8_weight_scale, p.fp8_channel_scales};
    else
      m.data = p.bf16;
    if (!m.data || !(m.alpha > 0.0F) || !std::isfinite(m.alpha)) return GW_OK;      // the plans report what is wrong
  }
  if (!stream_aligned(q)) return GW_OK;
  for (int i = 0; i < (second ? 2 : 1); ++i)
    if (!with.maps[i].get(kind, *matrix[i], with.plan.physical_n, q.k, &error))
      return fail(GW_CUDA_ERROR, "weight descriptor: " + error);
  q.ld_out = first.output;
  q.workspace = workspace;
  q.counters = counters;
  q.error = device_error_word();
  for (uint32_t row = 0; row < rows; row += kStreamMaxRows) {
    q.rows = std::min(rows - row, kStreamMaxRows);
    q.reread = rows - row > kStreamMaxRows;
    q.weights_settled = weights_settled || row != 0;      // of this projection's launches only the first follows another's
    q.input = static_cast<const bf16*>(input) + size_t(row) * q.k;
    q.output = static_cast<bf16*>(output) + size_t(row) * q.ld_out;
    GW_CUDA_CHECK(launch_stream(q, with.plan, with.maps[0], with.maps[1], s), "weight-streaming projection");
  }
  *done = true;
  return GW_OK;
}

namespace {
// 33 to 128 rows on the CTA pairs instead of the swap form, whose partial tiles go through global memory and take longer the more
// columns they have.  In passes of a graph, us with the quantiser, swap form / pairs, where one wave of wide tiles holds all channels:
//   FP8   64 x 5376x2048 11.2 / 9.4, 21504x5376 30.5 / 26.4; with few K slabs only beyond 64 rows (2816x4096 64 rows 8.8 / 9.2, 65
//         10.3 / 9.2); 128 x 2816x2816 11.4 / 9.4, 8192x2816 17.9 / 12.8
//   BF16  33 x 2816x2816 10.4 / 9.2; 128 x 5376x2048 17.1 / 12.3, 21504x5376 52.2 / 42.0
//   both  more than a third of the pairs' channels, 5376x8192 65 rows FP8 15.4 / 15.6, BF16 22.2 / 20.5, 128 rows 16.9 / 15.8, 23.9 / 20.8
//   NVFP4, whose tile is 256 rows high whatever their number, long K and few channels: 65 x 8192x2816 13.9 / 11.9, 12288x4096 16.6 /
//         16.2, 128 rows 15.0 / 12.9, 20.1 / 17.9; but 65 x 8192x5376 14.0 / 14.6, 112 x 4096x2816 10.7 / 11.9;
//         33 x 8192x2816 12.0 / 10.9, 8192x3072 11.9 / 11.0, 12288x2048 12.5 / 12.2, but 16384x2816 14.5 / 14.5, 21504x512 14.1 / 14.5
// Weights that the launch before wrote, more of them than L2 holds, stay on the swap form (MLP 5376 -> 21504 with dequantised weights
// 36 rows 286 / 292, 128 rows 312 / 312; 2816 -> 8192 86 / 84, 97 / 88).
// The pairs' sums are of more and shorter parts of K; the error against FP64 is no larger at any of these sizes.
constexpr size_t kBeyondL2 = size_t(126) << 20;
bool small_on_pairs(const DenseTuning& tuning, const DenseProblem& q) {
  if (!tuning.streams() || tuning.no_pair || q.rows <= 32) return false;
  const int channel_tiles = int((q.n + 255) / 256), pairs = sm_count() / 2;
  if (q.kind == GemmKind::nvfp4)
    return q.k >= 8192 && (q.rows > 64 ? channel_tiles <= pairs / 4 : channel_tiles <= pairs / 6 && q.k <= 12288) && q.n % 8 == 0 && reinterpret_cast<uintptr_t>(q.output) % 16 == 0;
  if (q.weights_fresh && size_t(q.n) * q.k * sizeof(bf16) > kBeyondL2) return false;
  return channel_tiles <= (q.rows <= 96 ? pairs / 3 : pairs / 2) && (q.kind == GemmKind::bf16 || q.rows > 64 || q.k >= 4096);
}
}  // namespace

gw_status launch_dense(const DenseProblem& q, DenseDescriptors* cache, cudaStream_t stream) {
  const DenseTuning& tuning = cache->tuning;
  // NVFP4 outputs may lie on any 2-byte boundary.  The swap form stores two bytes at a time, all other kernels sixteen.
  const bool unaligned = q.kind == GemmKind::nvfp4 && reinterpret_cast<uintptr_t>(q.output) % 16 != 0;
  const bool small_pairs = q.rows <= 128 && small_on_pairs(tuning, q);
  const bool swap = unaligned || (!small_pairs && dense_uses_swap_form(tuning, q.rows));
  const int block_n = small_pairs ? 256 : swap ? swap_block_n(q.rows) : dense_block_n(tuning, q.rows);
  if (cache->small_pairs != small_pairs || cache->swap != swap) {          // another route's maps have other boxes
    cache->small_pairs = small_pairs;
    cache->swap = swap;
    cache->weight = cache->activations = nullptr;
  }
  const bool fp4 = q.kind == GemmKind::nvfp4;
  const uint64_t row_bytes = fp4 ? q.k / 2 : (q.kind == GemmKind::bf16 ? uint64_t(2) * q.k : q.k);
  std::string error;
  // FP8 and BF16 beyond the swap form's rows, narrow ones too (BF16, K 2816, N 128, us, CTA pairs / single CTAs with 128- and
  // 256-wide tiles: 129 rows 11.5 / 13.2 / 15.6, 777 rows 11.7 / 13.5 / 16.2, 8192 rows 13.9 / 14.2 / 17.8; N 512 129 rows 12.1 /
  // 13.7 / 20.6).  Outputs of these kinds are 16-byte aligned and a multiple of 8 wide (plan creation and the run check it).
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
  // NVFP4 prefill: the CTA-pair kernel (each CTA stages half of the weight tile) unless disabled; also where one pair tile holds
  // all rows (us, with the quantiser, single CTAs / pairs: 130x2816x4096 13.8 / 10.7, 200x5376x16384 24.5 / 19.8, MLP of 200 rows
  // 117 / 84).
  if (fp4 && single_box && !tuning.no_pair) {
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
    params.weights_settled = q.weights_settled ? 1 : 0;
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
    const int stages = gemm_tc_k_stages(q.kind, GemmEpilogue::swap_store, row_bytes);
    const int split_grid = swap_split_grid(q.kind, params.total_work, stages, block_n);
    if (split_grid > 0) {
      params.split_counters = cache->split_counters;
      params.split_partials = static_cast<float*>(q.split_workspace);
      grid = split_grid;
    }
  }
  GW_CUDA_CHECK(launch_gemm_tc(q.kind, swap ? GemmEpilogue::swap_store : GemmEpilogue::direct_store, block_n, params,
                               grid, stream),
                fp4 ? "NVFP4 tensor-core GEMM" : (q.kind == GemmKind::bf16 ? "BF16 tensor-core GEMM" : "FP8 tensor-core GEMM"));
  return GW_OK;
}

// Beyond the swap form's rows always; with fewer where one wave of pair tiles (NVFP4: half of one) holds all channels, so that
// three launches stand against the swap form's four to nine.  MLP of joined gate and up, us launched one by one | in a graph, swap form /
// this:
//   NVFP4 16x2816 -> 4096 21.8 / 20.5 | 17.1 / 19.2, 128x2048 -> 4096 22.6 / 21.6 | 21.3 / 20.5; with few channels for their K slower either
//         way, 96x5376 -> 2048 22.2 / 24.3 | 20.5 / 23.2; 40x4096 -> 8192 27.2 / 29.7
//   FP8   16x2816 -> 4096 22.0 / 20.3 | 16.5 / 18.9, 64x2816 -> 4096 22.6 / 21.2 | 21.4 / 19.9; apart 16x2816 -> 2176 - | 24.3 / 14.6
//   BF16  64x2816 -> 4096 29.3 / 25.7 | 28.6 / 24.8; up to 32 rows slower, 16x2816 -> 2176 20.9 / 22.3 | 20.5 / 21.1, 16x5376 -> 2048
//         25.7 / 30.3 | 25.2 / 29.3, and up to 64 with few channels for their K, 48x5376 -> 2048 29.3 / 31.4 | 28.9 / 30.5
//
// NVFP4 of few rows has one accumulator here (tensor memory is full beside the scales), so it stays on the swap form where that
// divides K: the sums would be of longer parts, and with widely varying block scales further from the exact ones (outputs of an MLP
// that differ from those with exact gate and up, 16x5376 -> 2048: none / 2.7e-3).
bool dense_geglu_pays(const DenseTuning& tuning, GemmKind kind, uint32_t rows, uint32_t k, uint32_t n) {
  if (tuning.form != 0 || tuning.block_n != 0 || tuning.no_pair) return false;
  if (!dense_uses_swap_form(tuning, rows)) return true;
  const bool few_channels = 2 * size_t(n) < k;
  if (kind == GemmKind::bf16 && (rows <= 32 || (rows <= 64 && few_channels))) return false;
  if (kind == GemmKind::nvfp4) {
    if (few_channels) return false;
    const int tiles = int((n + 127) / 128), stages = gemm_tc_k_stages(kind, GemmEpilogue::swap_store, k / 2);
    for (const int of : {tiles, 2 * tiles})          // gate and up apart, joined
      if (swap_split_grid(kind, of, stages, swap_block_n(rows)) > 0) return false;
  }
  return rows > 8 && int((n + 127) / 128) <= sm_count() / (kind == GemmKind::nvfp4 ? 4 : 2);
}

gw_status launch_dense_geglu(const GegluProblem& q, DenseDescriptors* cache, cudaStream_t stream) {
  std::string error;
  const uint32_t physical = (q.n + 127) / 128 * 128;
  const void* from[3] = {q.activations, q.weight[0], q.weight[1]};
  for (int i = 0; i < 3; ++i)
    if (cache->geglu_from[i] != from[i]) {
      if (!encode_tensor_map_2d(&cache->geglu_maps[i], from[i], q.k / 2, i == 0 ? q.rows : physical, 128, &error))
        return fail(GW_CUDA_ERROR, "gate/up descriptor: " + error);
      cache->geglu_from[i] = from[i];
    }
  PairGemmParams pair{};
  pair.map_tokens = cache->geglu_maps[0];
  pair.map_weights = cache->geglu_maps[1];
  pair.map_up = cache->geglu_maps[2];
  pair.sf_tokens = q.activation_scales;
  pair.token_row_blocks = int32_t((q.rows + 127) / 128);
  pair.k = int32_t(q.k);
  pair.rows = int32_t(q.rows);
  pair.n = int32_t(q.n);
  pair.l_tiles = int32_t((q.rows + 255) / 256);
  pair.c_tiles = int32_t(physical / 128);
  pair.out = q.packed;
  pair.scales_out = q.scales;
  pair.alpha = q.alpha[0];
  pair.alpha_up = q.alpha[1];
  pair.inverse_scale = q.inverse_scale;
  for (int i = 0; i < 2; ++i) pair.sf_gate_up[i] = q.weight_scales[i];
  pair.error = q.error;
  GW_CUDA_CHECK(launch_gemm_pair_geglu(pair, sm_count(), stream), "NVFP4 CTA-pair gate/up GEMM with GeGLU + quantise");
  return GW_OK;
}

gw_status launch_dense_geglu_wide(const WideGegluProblem& q, DenseDescriptors* cache, cudaStream_t stream) {
  std::string error;
  const uint64_t row_bytes = q.kind == GemmKind::bf16 ? uint64_t(2) * q.k : q.k;
  if (cache->geglu_wide.tile_rows == 0) cache->geglu_wide = pair_wide_tiles(q.rows, 2 * q.n, 0, sm_count());
  const void* from[3] = {q.activations, q.weight[0], q.weight[1]};
  for (int i = 0; i < 3; ++i)
    if (cache->geglu_from[i] != from[i]) {
      if (!encode_tensor_map_2d(&cache->geglu_maps[i], from[i], row_bytes, i == 0 ? q.rows : q.n, i == 0 ? uint32_t(cache->geglu_wide.tile_rows / 2) : 64, &error))
        return fail(GW_CUDA_ERROR, "gate/up descriptor: " + error);
      if (i == 0 && !encode_tensor_map_2d(&cache->geglu_piece_map, from[0], row_bytes, q.rows, uint32_t(cache->geglu_wide.piece_rows / 2), &error))
        return fail(GW_CUDA_ERROR, "gate/up descriptor: " + error);
      cache->geglu_from[i] = from[i];
    }
  PairWideParams pair{};
  pair.map_tokens = cache->geglu_maps[0];
  pair.map_piece = cache->geglu_piece_map;
  pair.map_weights = cache->geglu_maps[1];
  pair.map_up = cache->geglu_maps[2];
  pair.k_stages = int32_t((row_bytes + 127) / 128);
  pair.last_kb = int32_t((row_bytes - uint64_t(pair.k_stages - 1) * 128 + 31) / 32);
  pair.rows = int32_t(q.rows);
  pair.n = int32_t(q.n);
  pair.tiles = cache->geglu_wide;
  pair.out = q.output;
  pair.ld_out = q.n;
  pair.alpha = q.alpha[0];
  pair.alpha_up = q.alpha[1];
  pair.channel_alpha = q.channel_alpha[0];
  pair.channel_alpha_up = q.channel_alpha[1];
  pair.inverse_scale = q.inverse_scale;
  pair.error = q.error;
  GW_CUDA_CHECK(launch_gemm_pair_wide_geglu(q.kind == GemmKind::fp8, q.inverse_scale != 0.0F, pair, sm_count(), stream),
                "CTA-pair gate/up GEMM with GeGLU");
  return GW_OK;
}

}  // namespace gw
