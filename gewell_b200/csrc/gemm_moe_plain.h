// Launch functions of the grouped FP8 and BF16 GEMMs of MoE layers whose experts are all of one kind (gemm_moe_plain.cu): an
// expert's token rows on the columns, `tile_rows` (64 or 128) at a time.  FP8 experts must quantise the gate and up inputs
// with one scale.
#pragma once

#include "gemm_pair_moe.h"

namespace gw {

// params.kind: kMoeKindFp8 or kMoeKindBf16; map_tokens: token rows in that type, box of tile_rows rows.  Gate/up writes both
// BF16 captures and, FP8, the down input to packed_out ([capacity, 704]); the activated capture is BF16's down input.  Both read
// the offsets and the weights before they wait for the kernel in front of them: that one belongs to the same call and writes
// neither.
cudaError_t launch_moe_plain_gate_up(int tile_rows, const PairMoeParams& params, int sm_count, cudaStream_t stream);
cudaError_t launch_moe_plain_down(int tile_rows, const PairMoeParams& params, int sm_count, cudaStream_t stream);

}  // namespace gw
