// Grouped GEMM of token rows with the expert weights on the M side of a CTA pair (ragged_gemm.cu): forward and data-gradient
// modes of GemmArgs (kFwd1, kFwd2, kDgrad1, kPlain; args.ctas = 2), with or without the fused transport.
#pragma once

#include "grouped_gemm.h"

namespace epb {

// tmW: kFwd1 make_tmap_gate_up, kDgrad1 make_tmap_blocks (N % 64 == 0), else K-major weights, box {64 k, 128, 1}; tmX: token rows,
// 2-D, box {64 k, 128}.
cudaError_t launch_ragged_gemm(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmArgs& args, int num_sms,
                               cudaStream_t stream);

}  // namespace epb
