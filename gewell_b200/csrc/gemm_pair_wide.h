// Launch description of the CTA-pair prefill GEMM for FP8 and BF16 weights (gemm_pair_wide.cu):
// Y[rows, n] = bf16(alpha * X . W^T), output channels on the lanes (256 per pair tile), tokens on the columns
// (tile_rows per tile, half of them staged by each CTA of the pair).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace gw {

// Division of [token tiles x channel tiles] over the pairs.
struct PairWideTiles {
  int32_t tile_rows = 0;           // token columns per tile (0: not computed yet)
  int32_t channel_tiles, token_tiles;
  int32_t whole;                   // tiles that are taken whole: as many as fill waves of all pairs
  int32_t pieces, piece_rows;      // of each tile behind them: how many pieces, and their token columns
  int32_t split = 0;               // split form, one tile per cluster: pairs that share its K loop
};

struct PairWideParams {
  CUtensorMap map_weights;         // weights [n, k], box 128 rows x 128 bytes, 128-byte swizzle
  CUtensorMap map_tokens;          // activations [rows, k], box tile_rows / 2 rows
  CUtensorMap map_piece;           // the same, box piece_rows / 2 rows
  int32_t k_stages;                // 128-byte slabs of K
  int32_t last_kb;                 // 32-byte K blocks in the last one
  int32_t rows, n;
  PairWideTiles tiles;
  int32_t stages, stage_bytes;     // of the operand ring (set by the launch)
  void* out;                       // BF16 [rows, ld_out], 16-byte aligned rows
  int64_t ld_out;
  float alpha;
  const float* channel_alpha;      // optional multiplier per output channel instead of alpha
  // launch_gemm_pair_wide_geglu: map_weights (box 64 rows) and the multipliers above are the gate's, these the up projection's
  CUtensorMap map_up;
  float alpha_up, inverse_scale;   // inverse_scale: 1 / input scale of the FP8 projection that takes the result
  const float* channel_alpha_up;
  uint32_t* error;
};

// The division for this shape that takes least: `n` channels, 256 per tile; k_stages != 0: the split form is possible, and for at most
// 128 rows it is what is taken (which needs one wave of tiles).
PairWideTiles pair_wide_tiles(uint32_t rows, uint32_t n, int k_stages, int sm_count);

// GeGLU of two projections with n channels each, as BF16 [rows, n] or (`quantise`) E4M3 [rows, n].  n is a multiple of 64, a tile
// has 128 channels of each.
cudaError_t launch_gemm_pair_wide_geglu(bool fp8, bool quantise, const PairWideParams& params, int sm_count, cudaStream_t stream);

cudaError_t launch_gemm_pair_wide(bool fp8, const PairWideParams& params, int sm_count, cudaStream_t stream);

}  // namespace gw
