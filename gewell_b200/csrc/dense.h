// One dense projection Y[rows, n] = bf16(alpha * Xq . Wq^T) on the tcgen05
// kernel: picks the operand roles and tile for the row count, builds the TMA
// descriptors (cached per plan) and launches.
#pragma once

#include <map>
#include <tuple>
#include <utility>
#include <vector>

#include "common.cuh"
#include "decode_stream.h"
#include "gemm_pair_wide.h"
#include "gemm_tc.cuh"

namespace gw {

// Tuning overrides of the dense projections, read from the environment once per plan (when its
// descriptors are first used), not at every call:
//   GW_DENSE_FORM=swap|direct, GW_DENSE_BLOCK_N=128|256   operand roles / column tile
//   GW_DENSE_NO_PAIR=1    projections of many rows stay on the single-CTA kernel
//   GW_DENSE_NO_SPLIT=1   decode-shaped plans run whole tiles per CTA
// Each of them but the third also keeps small row counts off the weight-streaming kernel.
struct DenseTuning {
  char form = 0;            // 's', 'd' or 0
  int block_n = 0;
  bool no_pair = false, no_split = false;
  bool streams() const { return form == 0 && block_n == 0 && !no_split; }
  static DenseTuning from_environment();
};

struct DenseDescriptors {          // re-encoded only when a pointer changes
  DenseTuning tuning = DenseTuning::from_environment();
  const void* weight = nullptr;
  const void* activations = nullptr;
  const void* weight_scales = nullptr;
  CUtensorMap weight_map{}, activation_map{}, weight_scale_map{};
  bool small_pairs = false, swap = false;          // which route the maps are for
  const void* weight_half = nullptr;
  CUtensorMap weight_half_map{};     // 128-row box over the weights (CTA-pair kernel: each CTA stages half a tile)
  PairWideTiles wide;                // FP8 / BF16 CTA-pair kernel: division of the work
  CUtensorMap piece_map{};           // and its box over the activations for the pieces of tiles
  // the GeGLU forms (launch_dense_geglu, launch_dense_geglu_wide): division; the activations (and pieces of them), gate and up
  PairWideTiles geglu_wide;
  CUtensorMap geglu_piece_map{};
  const void* geglu_from[3] = {};
  CUtensorMap geglu_maps[3]{};
  // Split mode: one arrival counter per weight tile, owned by the plan (device memory,
  // zeroed at creation; the kernel leaves every counter at zero again).
  int32_t* split_counters = nullptr;
  // Small row counts: how the weight-streaming kernel divides the work (its counters are split_counters).
  StreamPlan stream;
  StreamMaps stream_maps;
  cudaError_t allocate_split_counters(GemmKind kind, uint32_t rows, uint32_t k, uint32_t n);
  // Scratch for FP32 partial sums of either form (0: none), once the counters exist.
  size_t split_bytes(uint32_t rows) const;
  ~DenseDescriptors();
};

struct DenseProblem {
  GemmKind kind;
  uint32_t rows, k, n;
  const void* weight;              // [n, k] E4M3, [n, k/2] packed E2M1 or [n, k] BF16
  const uint8_t* weight_scales;    // NVFP4 only
  const void* activations;         // quantised [rows, k(/2)], or the BF16 input itself for the BF16 kind
  const uint8_t* activation_scales;
  float alpha;
  const float* channel_alpha;
  void* output;
  uint32_t* error;
  // Optional, decode shapes only: dense_split_bytes() bytes, 256-byte aligned, for FP32
  // partial tiles.  With it (and the plan's counters) the K loop of the weight tiles is
  // divided evenly over the SMs (see GemmParams).
  void* split_workspace = nullptr;
  // In front of this launch, or of the quantiser of its activations, the same call launched a kernel that does not write the
  // weights: the swap form reads its first weight tiles while that kernel still runs.  Otherwise they wait in L2 meanwhile.
  bool weights_settled = false;
  // The launch in front of this one wrote the weights (the dequantiser of the BF16 path).
  bool weights_fresh = false;
};

// true: weights on the 128-lane operand and tokens on the column operand.
bool dense_uses_swap_form(const DenseTuning& tuning, uint32_t rows);
int dense_block_n(const DenseTuning& tuning, uint32_t rows);

// Bytes of split workspace a projection of so many rows can use (0: none).
size_t dense_split_bytes(const DenseTuning& tuning, uint32_t rows);

// Whether the weight-streaming kernel is the faster one for this shape (n: output channels of all matrices together).
bool stream_pays(StreamKind kind, const StreamPlan& plan, uint32_t rows, uint32_t k, size_t n);

// The problem on the weight-streaming kernel; *done = false when its pointers keep it off that kernel.
gw_status launch_dense_stream(const StreamProblem& problem, DenseDescriptors* cache, cudaStream_t stream, bool* done);

// The weight-streaming launches of an object whose projections run one after another: plans by (kind, K, physical N,
// two matrices) for the row count of the last prepare(), the counters they share, and the tensor maps of the last
// matrices under each key.
struct StreamBook {
  using Key = std::tuple<int, uint32_t, uint32_t, bool>;
  struct Entry { StreamPlan plan; StreamMaps maps[2]; };
  std::map<Key, Entry> entries;
  int32_t* counters = nullptr;
  size_t counter_bytes = 0;
  uint32_t rows = 0;
  StreamBook() = default;
  StreamBook(const StreamBook&) = delete;
  StreamBook& operator=(const StreamBook&) = delete;
  ~StreamBook();
  // What another row count needs, built beside what run() uses; publish() puts it in its place and cannot fail, so that an
  // object publishes all of its parts or none.  shapes: (K, physical N); `workspace_bytes`: of the workspace that run() will
  // be given.
  struct Staged {
    std::map<Key, Entry> entries;
    int32_t* counters = nullptr;       // larger ones, where the present ones do not suffice
    size_t counter_bytes = 0;
    uint32_t rows = 0;
    Staged() = default;
    Staged(const Staged&) = delete;
    Staged& operator=(const Staged&) = delete;
    ~Staged();
  };
  gw_status stage(uint32_t rows, const std::vector<std::pair<uint32_t, uint32_t>>& shapes, size_t workspace_bytes, Staged* staged) const;
  void publish(Staged* staged);
  // The projection `first` -- or, with `second`, GeGLU of both -- into [rows, first.output]; *done = false when the shape,
  // the storage or the pointers keep it off the kernel.
  gw_status run(const gw_projection& first, const gw_projection* second, const void* input, void* output, bool fp4, void* workspace,
                bool weights_settled, cudaStream_t stream, bool* done);
};

gw_status launch_dense(const DenseProblem& problem, DenseDescriptors* cache, cudaStream_t stream);

// GeGLU of two projections of the same rows, quantised for the projection that takes it, in one launch.
struct GegluProblem {
  uint32_t rows, k, n;                       // n: channels of each projection; their matrices have whole 128-row tiles
  const uint8_t *weight[2], *weight_scales[2];   // gate, up
  float alpha[2];
  const uint8_t *activations, *activation_scales;
  float inverse_scale;                       // 1 / input scale of the projection that takes the result
  uint8_t *packed, *scales;                  // [rows, n / 2] and its tiled scales
  uint32_t* error;
};
// Whether that is the faster way for gate and up projections of n channels each.
bool dense_geglu_pays(const DenseTuning& tuning, GemmKind kind, uint32_t rows, uint32_t k, uint32_t n);
gw_status launch_dense_geglu(const GegluProblem& problem, DenseDescriptors* cache, cudaStream_t stream);

// The same of FP8 or BF16 projections; the result is E4M3 (inverse_scale != 0) or BF16.
struct WideGegluProblem {
  GemmKind kind;
  uint32_t rows, k, n;
  const void *activations, *weight[2];       // gate, up
  float alpha[2];
  const float* channel_alpha[2];
  float inverse_scale;                       // 1 / input scale of the FP8 projection that takes the result, or 0
  void* output;                              // [rows, n]
  uint32_t* error;
};
gw_status launch_dense_geglu_wide(const WideGegluProblem& problem, DenseDescriptors* cache, cudaStream_t stream);

// gw_*_plan_run as a step of a longer call (api.cu): `weights_settled`, `weights_fresh` as in DenseProblem.  The public entry points pass
// false.
gw_status run_nvfp4_plan(gw_nvfp4_plan* plan, const void* input, const uint8_t* weight_data, const uint8_t* weight_scales, float input_scale,
                         float weight_scale, void* output, void* scratch, size_t scratch_capacity, cudaStream_t stream, int transform,
                         bool weights_settled);
gw_status run_fp8_plan(gw_fp8_plan* plan, const void* input, const uint8_t* weight_data, float input_scale, float weight_scale,
                       const float* channel_scales, void* output, void* scratch, size_t scratch_capacity, cudaStream_t stream, int transform,
                       bool weights_settled);
gw_status run_bf16_plan(gw_bf16_plan* plan, const void* input, const void* weight, void* output, void* scratch, size_t scratch_capacity,
                        cudaStream_t stream, bool weights_settled, bool weights_fresh = false);

// Gate, up, GeGLU and the quantiser of `down` into `buffer` (packed rows and their tiled scales, as in a plan's
// scratch), then down over them; *done = false when shape, storage or pointers keep the three off that way.  `gate_plan`,
// `down_plan`: of the gate's and of down's shape; `buffer`: room for BF16 [rows, n], n = down.input.
gw_status run_nvfp4_geglu(gw_nvfp4_plan* gate_plan, gw_nvfp4_plan* down_plan, const gw_projection& gate, const gw_projection& up,
                          const gw_projection& down, const void* input, void* buffer, void* output, void* scratch, size_t scratch_capacity,
                          cudaStream_t stream, bool* done);

// GeGLU of FP8 or BF16 gate and up projections of a prefill pass into `product`: E4M3 for `down_plan` and `down` where that is FP8, and
// *packed = true, else BF16.  *done = false when shape, storage or pointers keep them off that way.  run_fp8_plan_packed, with the same
// scratch, runs down over the former.
gw_status run_fp8_geglu(gw_fp8_plan* gate_plan, const gw_projection& gate, const gw_projection& up, const gw_projection& down, const void* input,
                        void* product, void* scratch, size_t scratch_capacity, cudaStream_t stream, bool* packed, bool* done);
gw_status run_bf16_geglu(gw_bf16_plan* gate_plan, const gw_projection& gate, const gw_projection& up, const gw_projection& down,
                         const void* input, void* product, cudaStream_t stream, bool* packed, bool* done);
gw_status run_fp8_plan_packed(gw_fp8_plan* plan, const void* packed, const gw_projection& p, void* output, void* scratch,
                              size_t scratch_capacity, cudaStream_t stream);

// gw_projection_workspace_run on a stream of the caller's choice (projection.cu).
gw_status projection_workspace_run_on(gw_projection_workspace* workspace, const gw_projection* projection, const void* input, void* output,
                                      cudaStream_t stream, bool weights_settled);
// product = GeGLU of both projections of a prepared workspace in one launch; *done = false when that is not the faster
// way here.
gw_status projection_workspace_run_geglu(gw_projection_workspace* workspace, const gw_projection& gate, const gw_projection& up,
                                         const void* input, void* product, cudaStream_t stream, bool weights_settled, bool* done);
// Gate, up, GeGLU and down of a prepared workspace by run_nvfp4_geglu; `buffer`: BF16 [rows, down.input].
gw_status projection_workspace_run_mlp(gw_projection_workspace* workspace, const gw_projection& gate, const gw_projection& up,
                                       const gw_projection& down, const void* input, void* buffer, void* output, cudaStream_t stream, bool* done);

}  // namespace gw
