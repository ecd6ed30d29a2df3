// Block-scaled fp8 grouped GEMM for few rows per expert (narrow_gemm_fp8.cu): weights on the M side, token rows on the N side.
#pragma once

#include "grouped_gemm_fp8.h"

namespace epb {

constexpr int kNarrowFp8BoxRows = 32;  // token rows of one TMA box

// Batches with fewer routed units per weight slot than this take the narrow kernel: with few rows the 256-row tiles of the
// pair kernel are mostly padding.  Measured, both GEMMs with the activation in us, pair / narrow, rows per expert spread by a
// lognormal of 0.35 around the mean:
//   hidden x ffn x experts   16 rows     96 rows     128 rows    160 rows    191 rows    256 rows
//   7168 x 2048 x  32        321 / 252   341 / 267   344 / 307   374 / 403   385 / 441   469 / 521
//   5120 x 1536 x  40        228 / 183   242 / 212   247 / 221   260 / 271   292 / 307   353 / 375
//   2048 x  768 x 128        210 / 142   202 / 161   214 / 180   228 / 204   249 / 236   284 / 284
//   2048 x 1408 x  64        167 / 116   166 / 135   175 / 149   191 / 168   203 / 183   232 / 219
//   1024 x  512 x 256        161 / 119   184 / 172   195 / 191   206 / 209   224 / 234   246 / 274
// Up to 128 rows the narrow kernel wins everywhere; from there to the line each kernel wins by up to 14 % at some shapes, and
// by 384 rows the pair kernel is ahead at all of them.  (Pair before its stages of two k-blocks, which took 6 % off
// a prefill of 1024 rows an expert.)  (16 rows of the first shape read 1.41 GB of weights: 215 us at the rate
// of a copy.)
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
