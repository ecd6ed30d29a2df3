// Gradient of the mean token cross-entropy in one pass: log-probabilities in (fp32), bf16 gradient out, 6 bytes a value.
// The library chain it replaces fills and scatters the gradient of the log-probabilities (4 bytes), turns it into that of
// the fp32 logits (12) and casts it (6).  4096 x 32000: 570 us of kernels before, about 130 now (a GPT step 7145 -> 6733).
// Bound by HBM; one CTA per row, 32 bytes in and 16 out per thread and step.
#include "loss.h"

#include <cuda_bf16.h>

namespace epb {
namespace {

constexpr int kThreads = 512;

__global__ void __launch_bounds__(kThreads) cross_entropy_backward_kernel(CrossEntropyGradArgs a) {
  const int r = blockIdx.x, n_vec = a.vocab / 8;
  const float4* lp = reinterpret_cast<const float4*>(a.log_prob + (size_t)r * a.vocab);
  uint4* g = reinterpret_cast<uint4*>(a.grad) + (size_t)r * n_vec;
  const int64_t t = a.targets[r];
  const float scale = t == kIgnoreIndex ? 0.f : *a.grad_out / *a.weight;
#pragma unroll 2
  for (int v = threadIdx.x; v < n_vec; v += kThreads) {
    const float4 lo = lp[2 * v], hi = lp[2 * v + 1];
    const float f[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    const int hit = (t >> 3) == v ? (int)(t & 7) : -1;
    uint4 o;
    __nv_bfloat162* po = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float a0 = expf(f[2 * j]) * scale - (2 * j == hit ? scale : 0.f);
      const float a1 = expf(f[2 * j + 1]) * scale - (2 * j + 1 == hit ? scale : 0.f);
      po[j] = __floats2bfloat162_rn(a0, a1);
    }
    g[v] = o;
  }
}

}  // namespace

cudaError_t launch_cross_entropy_backward(const CrossEntropyGradArgs& a, cudaStream_t stream) {
  if (a.rows < 0 || a.vocab <= 0 || a.vocab % 8 != 0) return cudaErrorInvalidValue;
  if (a.rows > 0) cross_entropy_backward_kernel<<<a.rows, kThreads, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace epb
