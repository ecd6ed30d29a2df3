// Rotary embedding fused with the split of the packed projection: q and k are rotated (x1, x2 the halves of a head:
// x1 cos - x2 sin, x1 sin + x2 cos) and laid out per head, v stays where it is; the backward pass applies the transposed
// rotation and writes the packed gradient.  Bound by HBM, one read and one write of the activations per direction; the
// elementwise chain this replaces (slices, four products, sums, concatenations, layout copies, and their gradients) moved
// the q and k halves about ten times.  GPT step of 4096 tokens, 16 heads of 128: 6676 -> 6165 us with the same bits.
#include "rope.h"

#include <cuda_bf16.h>

#include "common.cuh"

namespace epb {
namespace {

__device__ __forceinline__ void load8(const void* p, float (&f)[8]) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void store8(void* p, const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = v;
}

__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// One thread: 8 elements of the first half of a head and their 8 partners of the second half, for q, k or (backward) v.
template <bool kBackward>
__global__ void __launch_bounds__(256) rope_kernel(RopeArgs a, __nv_bfloat16* packed) {
  const int half = a.dim / 2, vecs = half / 8;
  constexpr int kParts = kBackward ? 3 : 2;
  const long long total = (long long)a.B * a.S * kParts * a.heads * vecs;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int v = (int)(i % vecs);
  long long r = i / vecs;
  const int h = (int)(r % a.heads);
  r /= a.heads;
  const int which = (int)(r % kParts);
  r /= kParts;
  const int s = (int)(r % a.S), b = (int)(r / a.S);
  __nv_bfloat16* in = packed + ((((long long)b * a.S + s) * 3 + which) * a.heads + h) * a.dim + v * 8;
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(a.out[which]) + b * a.stride[which][0] + h * a.stride[which][1] +
                       s * a.stride[which][2] + v * 8;
  const __nv_bfloat16* src = kBackward ? out : in;
  __nv_bfloat16* dst = kBackward ? in : out;
  float x1[8], x2[8];
  load8(src, x1);
  load8(src + half, x2);
  if (which < 2) {
    float c[8], n[8];
    load8(reinterpret_cast<const __nv_bfloat16*>(a.cos) + (long long)s * half + v * 8, c);
    load8(reinterpret_cast<const __nv_bfloat16*>(a.sin) + (long long)s * half + v * 8, n);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sn = kBackward ? -n[j] : n[j];
      // the products are rounded to bf16 as the elementwise formulation rounds them
      const float y1 = round_bf16(x1[j] * c[j]) - round_bf16(x2[j] * sn), y2 = round_bf16(x1[j] * sn) + round_bf16(x2[j] * c[j]);
      x1[j] = y1;
      x2[j] = y2;
    }
  }
  store8(dst, x1);
  store8(dst + half, x2);
}

template <bool kBackward>
cudaError_t launch(const RopeArgs& a, void* packed, cudaStream_t stream) {
  if (a.dim <= 0 || a.dim % 16 != 0 || a.B < 0 || a.S < 0 || a.heads <= 0) return cudaErrorInvalidValue;
  for (int i = 0; i < (kBackward ? 3 : 2); ++i)
    for (int j = 0; j < 3; ++j)
      if (a.stride[i][j] % 8 != 0) return cudaErrorInvalidValue;
  const long long total = (long long)a.B * a.S * (kBackward ? 3 : 2) * a.heads * (a.dim / 16);
  if (total == 0) return cudaSuccess;
  if ((total + 255) / 256 > 0x7fffffffll) return cudaErrorInvalidValue;
  rope_kernel<kBackward><<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(a, reinterpret_cast<__nv_bfloat16*>(packed));
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_rope(const RopeArgs& a, cudaStream_t stream) { return launch<false>(a, const_cast<void*>(a.qkv), stream); }
cudaError_t launch_rope_backward(const RopeArgs& a, void* grad_qkv, cudaStream_t stream) { return launch<true>(a, grad_qkv, stream); }

}  // namespace epb
