// Grouped GEMM for few rows per expert (narrow_gemm.cu): weights on the M side of the tensor core, token rows on its N
// side.  The inference forward's two GEMMs: GemmArgs of grouped_gemm.h with mode kFwd1 (with or without the fused transport;
// out0 null, the pre-activations are not kept) or kFwd2.
#pragma once

#include "grouped_gemm.h"

namespace epb {

constexpr int kNarrowBoxRows = 32;  // token rows of one TMA box: box of the token map {64 k, kNarrowBoxRows}

// Inference batches with at most this many routed units per weight slot take the narrow kernel.  Measured, GEMM1 + GEMM2 in us,
// wide / narrow, rows per expert spread by a lognormal of 0.35 around the mean:
//   hidden x ffn x experts   4 rows       96 rows      128 rows     192 rows     384 rows
//   2048 x  768 x 128        327 /  212   351 /  254   353 /  260   381 /  322   629 /  536
//   5120 x 1536 x 160       1856 / 1176  2210 / 1397  2132 / 1867  2246 / 2312  3672 / 3808
//   2048 x 1408 x  64        302 /  206   295 /  241   311 /  268   337 /  337   570 /  578
// One line for every shape, at the most rows where the narrow kernel won each of them: the weights' bytes bound the launch up
// to there.  Beyond it the shapes disagree.  Wide rows and many weights do better on the full 256-row tiles, which move fewer
// operand bytes per flop; the first shape, with its short reductions, would keep 15 % on the narrow kernel up to 384 rows.
constexpr int kNarrowRowsPerSlot = 128;

// tmW: the weight map that grouped_gemm.h's kernels use as B (K-major box {64, 128, 1}); tmX: token rows, 2-D, box
// {64, kNarrowBoxRows}.
cudaError_t launch_narrow_gemm(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmArgs& args, int num_sms,
                               cudaStream_t stream);

}  // namespace epb
