// Grouped GEMM for few rows per expert (narrow_gemm.cu): weights on the M side of the tensor core, token rows on its N
// side.  The inference forward's two GEMMs: GemmArgs of grouped_gemm.h with mode kFwd1 (with or without the fused transport;
// out0 null, the pre-activations are not kept) or kFwd2.
#pragma once

#include "grouped_gemm.h"

namespace epb {

constexpr int kNarrowBoxRows = 32;  // token rows of one TMA box: box of the token map {64 k, kNarrowBoxRows}

// Inference batches with at most this many routed units per weight slot take the narrow kernel.  Measured, GEMM1 + GEMM2 in us,
// CTA pair (ragged_gemm.cu) / narrow, rows per expert spread by a lognormal of 0.35 around the mean, back to back:
//   hidden x ffn x experts   96 rows      128 rows     192 rows     384 rows
//   2048 x  768 x 128        248 /  232   264 /  265   302 /  331   476 /  554
//   5120 x 1536 x 160       1366 / 1252  1524 / 1514  1584 / 1936  2683 / 3780
//   2048 x 1408 x  64        258 /  241   267 /  341   289 /  369   409 /  576
// One line for every shape: below it the weights' bytes bound the launch and the narrow kernel moves fewer others, above it an
// expert's rows no longer fit one of its tiles.  At the line the two are level, but for the third shape under the power limit
// (by itself the narrow kernel takes 232-250 there).
constexpr int kNarrowRowsPerSlot = 128;

// tmW: the weight map that grouped_gemm.h's kernels use as B (K-major box {64, 128, 1}); tmX: token rows, 2-D, box
// {64, kNarrowBoxRows}.
cudaError_t launch_narrow_gemm(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmArgs& args, int num_sms,
                               cudaStream_t stream);

}  // namespace epb
