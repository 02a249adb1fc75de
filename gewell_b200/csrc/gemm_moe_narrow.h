// Launch functions of the grouped NVFP4 GEMMs of the MoE layer for batches whose experts get a few dozen rows each
// (gemm_moe_narrow.cu): an expert's token rows on the columns, `tile_rows` (64 or 128) at a time.  Experts must
// quantise the gate and up inputs with one scale.
#pragma once

#include "gemm_pair_moe.h"

namespace gw {

// params.map_tokens: box of tile_rows rows.  Both read the offsets and the weights before they wait for the kernel in front of
// them: that one belongs to the same call and writes neither.
cudaError_t launch_moe_narrow_gate_up(int tile_rows, const PairMoeParams& params, int sm_count, cudaStream_t stream);
cudaError_t launch_moe_narrow_down(int tile_rows, const PairMoeParams& params, int sm_count, cudaStream_t stream);

}  // namespace gw
