// Block-scaled fp8 building blocks shared by the fp8 grouped GEMMs: scale copies, the scaled MMA, its descriptors, and the
// power-of-two scales.
#pragma once

#include <cuda_fp8.h>

#include "common.cuh"

namespace epb {

// 512-byte scale chunk (32 rows x 16 B) -> 4 TMEM columns, replicated to the four 32-lane groups
__device__ __forceinline__ void tmem_cp_sf(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void umma_fp8_scaled(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                uint32_t sfa, uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%5], [%6], p;\n}\n"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
// Scale chunks: no swizzle, 8-row x 16-byte core matrices 128 B apart.
__device__ __forceinline__ uint64_t make_desc_sf(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(128 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}
// Instruction descriptor of the block-scaled kind: e4m3 x e4m3, both K-major, UE8M0 scales;
// sf ids select which of the four scale bytes of a TMEM word this MMA uses.
__device__ __forceinline__ uint32_t make_idesc_scaled(int n, int m, uint32_t a_sf_id, uint32_t b_sf_id) {
  return (b_sf_id << 4) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | ((uint32_t)(m >> 4) << 24) | (a_sf_id << 29);
}

// Power-of-two scale of a block with absolute maximum `amax`: the smallest 2^e with amax / 2^e <= 448.
__device__ __forceinline__ int scale_exponent(float amax) {
  if (!(amax > 0.f)) return -126;
  int ex;
  const float m = frexpf(amax * (1.f / 448.f), &ex);  // amax/448 = m * 2^ex, m in [0.5, 1)
  int e = (m == 0.5f) ? ex - 1 : ex;
  return max(-126, min(126, e));
}
__device__ __forceinline__ float exp2_int(int e) { return __int_as_float((e + 127) << 23); }  // e in [-126, 127]
__device__ __forceinline__ int chunk_byte(int r_in_128, int kb) { return (r_in_128 & 31) * 16 + (r_in_128 >> 5) * 4 + (kb & 3); }

}  // namespace epb
