// Block-scaled fp8 grouped GEMM for few rows per expert (narrow_gemm_fp8.cu): weights on the M side, token rows on the N side.
#pragma once

#include "grouped_gemm_fp8.h"

namespace epb {

constexpr int kNarrowFp8BoxRows = 32;  // token rows of one TMA box

// Batches with fewer routed units per weight slot than this take the narrow kernel: with few rows the 256-row tiles of the
// pair kernel are mostly padding.  (The line was drawn here for the single-CTA kernel that had these batches before.)
// 32 experts of 7168 x 2048, 16 rows each: both GEMMs 252 us and the activation pass 9 before, the whole decode step of a
// layer 364 -> 338 us (1.41 GB of weights: 212 us at the HBM rate).
constexpr int kNarrowFp8RowsPerSlot = 192;

struct NarrowFp8Args {
  Fp8GemmArgs g;           // N: output features (with q_out: F, and the weights hold gate rows then up rows); sfa: scales of the
                           // token rows, sfb: of the weights
  int w_box_rows;          // rows of a box of the weight map: 128 or 64
  // SwiGLU + 1 x 128 quantisation in the epilogue (both null: plain rows to g.out / g.out_ptrs)
  uint8_t* q_out;          // e4m3 [row_capacity, N]
  uint8_t* sf_out;         // its scale chunks
};

// tmW: e4m3 weights [slots, rows, K]; tmX: e4m3 token rows [row_capacity, K], box {128, kNarrowFp8BoxRows}.
cudaError_t launch_narrow_gemm_fp8(const CUtensorMap& tmW, const CUtensorMap& tmX, const NarrowFp8Args& args, int num_sms,
                                   cudaStream_t stream);

}  // namespace epb
