// Launch description of the weight-streaming projections for small row counts
// (decode_stream.cu): Y[rows, n] = bf16(alpha * Xq . Wq^T) for 1..8 rows (W4A16: 1..16), the
// activations quantised (or copied) by every thread block itself, every weight brought
// into shared memory once and contracted with warp-level tensor instructions.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <string>

namespace gw {

// w4a4: NVFP4 weights, activations quantised to NVFP4; w4a16: NVFP4 weights, BF16 activations;
// w8a8: E4M3 weights and activations; w16a16: BF16 both.
enum class StreamKind { w4a4, w4a16, w8a8, w16a16 };

constexpr uint32_t kStreamMaxRows = 16;   // W4A16; the other kinds take eight

struct StreamMatrix {
  const void* data = nullptr;            // [n, k] row-major, packed as the kind says
  const uint8_t* scales = nullptr;       // NVFP4: tiled E4M3 scales
  float alpha = 1.0F;                    // multiplier of the accumulator
  const float* channel_alpha = nullptr;  // FP8: optional multiplier per output channel, instead of alpha
};

struct StreamProblem {
  StreamKind kind;
  uint32_t rows, k, n;         // n: output channels to store (of each matrix when there are two)
  const void* input;           // BF16 [rows, k], or [rows, 2k] gate | up with gelu
  bool gelu = false;           // GeGLU of the input before it is quantised (w4a4, w8a8)
  float inverse_scale = 1.0F;  // 1 / input scale (w4a4, w8a8)
  uint8_t* packed = nullptr;          // w4a4, optional: the quantised activations, [rows, k / 2] ...
  uint8_t* packed_scales = nullptr;   // ... and their tiled scales (entries of rows that exist)
  StreamMatrix first, second;  // second.data != nullptr: gate and up, output = bf16 GeGLU of the two
  void* output;                // BF16 [rows, ld_out]
  size_t ld_out;
  void* workspace = nullptr;   // StreamPlan::workspace_bytes, 16-byte aligned
  int32_t* counters = nullptr; // StreamPlan::counter_count zeroed ints; left zero
  bool reread = false;         // another launch reads the same weights soon
  bool weights_settled = false;   // the same call launched the kernel before this one, which does not write the weights: the first
                                  // pieces are read while it still runs.  Otherwise they wait in L2 meanwhile
  uint32_t* error = nullptr;   // device error word
};

// How a problem of this shape is divided over the GPU.
struct StreamPlan {
  bool whole = false;          // every SM's range is whole row blocks: no sums to add up across SMs
  bool piece_sums = false;     // every piece of K is summed by itself
  bool usable = false;         // the shape can run here (widths a piece can walk, row count)
  uint32_t physical_n = 0;     // rows of each weight matrix in memory
  int tiles = 0;               // groups of eight token rows: 1 or 2
  int blocks = 0, chunks = 0, chunks_per_slab = 0, slabs = 0, grid = 0, max_units = 0;
  size_t workspace_bytes = 0;  // FP32 partial sums
  size_t counter_count = 0;
  size_t shared_bytes = 0;
  bool needs_workspace() const { return !whole; }
};
// `n`: rows of each weight matrix in memory; `pair`: two matrices.
StreamPlan plan_stream(StreamKind kind, uint32_t rows, uint32_t k, uint32_t n, bool pair, int sm_count);

// Tensor maps of one matrix, encoded again only when it changes.
struct StreamMaps {
  CUtensorMap weights{}, scales{};
  const void* data = nullptr;
  const void* scale_data = nullptr;
  bool get(StreamKind kind, const StreamMatrix& matrix, uint32_t n, uint32_t k, std::string* error);
};

// Pointers a launch needs beyond the plan: input and weights 16-byte aligned.
bool stream_aligned(const StreamProblem& problem);
cudaError_t launch_stream(const StreamProblem& problem, const StreamPlan& plan, const StreamMaps& first, const StreamMaps& second,
                          cudaStream_t stream);

}  // namespace gw
