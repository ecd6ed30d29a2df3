// Fused AdamW: one pass over parameter, gradient and both moments with 16-byte accesses.
// The expert weights of an MoE layer are one flat bf16 tensor per projection, so a single launch
// covers them; this replaces the multi-tensor optimizer launches over per-expert parameters.
#include "optim.h"

#include <cuda_bf16.h>

namespace epb {
namespace {

__device__ __forceinline__ void adam_one(float& p, float g, float& m, float& v, const AdamArgs& a) {
  p *= 1.f - a.lr * a.weight_decay;
  m = a.beta1 * m + (1.f - a.beta1) * g;
  v = a.beta2 * v + (1.f - a.beta2) * g * g;
  const float denom = sqrtf(v) / a.bias_correction2_sqrt + a.eps;
  p -= (a.lr / a.bias_correction1) * (m / denom);
}

// With a device step counter the two bias corrections are derived here.
__device__ __forceinline__ void resolve_step(AdamArgs& a) {
  if (a.step_ptr != nullptr) {
    const float t = (float)(*a.step_ptr);
    a.bias_correction1 = 1.f - powf(a.beta1, t);
    a.bias_correction2_sqrt = sqrtf(1.f - powf(a.beta2, t));
  }
}

// True while any status word of the guard is set (every thread reads the same few words; they are cached).
__device__ __forceinline__ bool guard_tripped(const AdamArgs& a) {
  if (a.guard == nullptr) return false;
  for (int i = 0; i < a.guard_rows; ++i)
    if (a.guard[4 * i] != 0) return true;
  return false;
}

// What every element of a step shares, computed once per block.
struct StepConst {
  float decay, step, inv_bc2, bc1, bc2;
  int fast;  // the error bound of update8 holds for these constants
};
__device__ __forceinline__ StepConst step_const(AdamArgs a) {
  resolve_step(a);
  StepConst c;
  c.decay = 1.f - a.lr * a.weight_decay;
  c.step = a.lr / a.bias_correction1;
  c.inv_bc2 = 1.f / a.bias_correction2_sqrt;
  c.bc1 = a.bias_correction1;
  c.bc2 = a.bias_correction2_sqrt;
  c.fast = a.eps >= 1e-15f && a.eps <= 1e5f && c.bc2 >= 1e-6f && c.bc2 <= 1.f && fabsf(c.step) <= 1e5f && fabsf(c.decay) <= 1e5f;
  return c;
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack2(uint32_t w) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w)); }
__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Eight weights.  The result has the bits of adam_one, at a third of its instructions: one IEEE square root and two IEEE
// divisions a weight kept the kernel at 5.5-6.2 TB/s.  A Ziv rounding test stands in for them (A. Ziv, "Fast evaluation of
// elementary mathematical functions with correctly rounded last bit", 1991): the update is taken with the approximate square
// root (relative error 2^-23) and division (2 ulp), so that it differs from adam_one's by less than 2^-20 of itself, plus
// half an ulp of the weight on either side for the last subtraction.  Where both ends of that interval round to the same bf16
// -- all but one weight in about ten thousand -- so does adam_one's value; the eight are redone by adam_one's formula
// otherwise, and where the denominator is out of the range of the bound (or not a number).
__device__ __forceinline__ void update8(uint4& pv, const float (&g)[8], uint4& mv, uint4& vv, const AdamArgs& a, const StepConst& c) {
  uint32_t* pp = reinterpret_cast<uint32_t*>(&pv);
  uint32_t* mp = reinterpret_cast<uint32_t*>(&mv);
  uint32_t* vp = reinterpret_cast<uint32_t*>(&vv);
  float m[8], v[8];
  uint32_t out[4], differ = 0u;
  bool redo = !c.fast;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 p2 = unpack2(pp[k]), m2 = unpack2(mp[k]), v2 = unpack2(vp[k]);
    float lo[2], hi[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = 2 * k + h;
      const float p = (h ? p2.y : p2.x) * c.decay;
      m[i] = a.beta1 * (h ? m2.y : m2.x) + (1.f - a.beta1) * g[i];
      v[i] = a.beta2 * (h ? v2.y : v2.x) + (1.f - a.beta2) * g[i] * g[i];
      const float denom = fmaf(sqrt_approx(v[i]), c.inv_bc2, a.eps);
      redo |= !(denom <= 1e10f);
      const float u = c.step * __fdividef(m[i], denom);
      const float q = p - u;
      const float margin = fmaf(fabsf(u), 0x1p-20f, fmaf(fabsf(q), 0x1p-23f, 1e-30f));  // 1e-30: results near zero are redone
      lo[h] = q - margin;
      hi[h] = q + margin;
    }
    out[k] = pack2(lo[0], lo[1]);
    differ |= out[k] ^ pack2(hi[0], hi[1]);
  }
  if (redo || differ != 0u) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float2 p2 = unpack2(pp[k]), m2 = unpack2(mp[k]), v2 = unpack2(vp[k]);
      adam_one(p2.x, g[2 * k], m2.x, v2.x, a);
      adam_one(p2.y, g[2 * k + 1], m2.y, v2.y, a);
      out[k] = pack2(p2.x, p2.y);
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    pp[k] = out[k];
    mp[k] = pack2(m[2 * k], m[2 * k + 1]);
    vp[k] = pack2(v[2 * k], v[2 * k + 1]);
  }
}

// One vector of eight weights a thread over a grid that covers the tensor: the loads of a block are in flight while its
// constants are computed, and the next blocks' while it stores.  A grid of 16 blocks per SM that strode over the tensor was
// 4-7 % slower.  Bound by HBM.  bf16 gradients (14 bytes a weight), before -> now: 940 M weights 6.14 -> 6.70 TB/s, 66 M
// 5.79 -> 6.50; fp32 gradients (16 bytes), 940 M: 6.38 -> 7.10.
__global__ void __launch_bounds__(256) adamw_bf16_kernel(AdamArgs a) {
  __shared__ StepConst shared;
  const size_t n_vec = a.numel / 8;
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint4* p4 = reinterpret_cast<uint4*>(a.param);
  uint4* m4 = reinterpret_cast<uint4*>(a.exp_avg);
  uint4* v4 = reinterpret_cast<uint4*>(a.exp_avg_sq);
  const bool have = i < n_vec;
  uint4 pv, mv, vv, g0, g1;
  if (have) {
    pv = p4[i];
    mv = m4[i];
    vv = v4[i];
    const uint4* gq = reinterpret_cast<const uint4*>(a.grad);
    g0 = gq[a.grad_f32 ? 2 * i : i];
    if (a.grad_f32) g1 = gq[2 * i + 1];
  }
  if (threadIdx.x == 0) shared = step_const(a);
  __syncthreads();
  if (guard_tripped(a)) return;
  const StepConst c = shared;
  a.bias_correction1 = c.bc1;
  a.bias_correction2_sqrt = c.bc2;
  if (have) {
    float g[8];
    if (a.grad_f32) {
      const uint32_t w[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) g[k] = __uint_as_float(w[k]);
    } else {
      const uint32_t w[4] = {g0.x, g0.y, g0.z, g0.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 t = unpack2(w[k]);
        g[2 * k] = t.x;
        g[2 * k + 1] = t.y;
      }
    }
    update8(pv, g, mv, vv, a, c);
    p4[i] = pv;
    m4[i] = mv;
    v4[i] = vv;
  } else if (i == n_vec) {
    // tail (numel not a multiple of 8)
    __nv_bfloat16* p1 = reinterpret_cast<__nv_bfloat16*>(a.param);
    const __nv_bfloat16* g1 = reinterpret_cast<const __nv_bfloat16*>(a.grad);
    __nv_bfloat16* m1 = reinterpret_cast<__nv_bfloat16*>(a.exp_avg);
    __nv_bfloat16* v1 = reinterpret_cast<__nv_bfloat16*>(a.exp_avg_sq);
    for (size_t j = n_vec * 8; j < a.numel; ++j) {
      float p = __bfloat162float(p1[j]), m = __bfloat162float(m1[j]), v = __bfloat162float(v1[j]);
      const float g = a.grad_f32 ? reinterpret_cast<const float*>(a.grad)[j] : __bfloat162float(g1[j]);
      adam_one(p, g, m, v, a);
      p1[j] = __float2bfloat16_rn(p);
      m1[j] = __float2bfloat16_rn(m);
      v1[j] = __float2bfloat16_rn(v);
    }
  }
}

__global__ void __launch_bounds__(256) adamw_f32_kernel(AdamArgs a) {
  if (guard_tripped(a)) return;
  resolve_step(a);
  float* p = reinterpret_cast<float*>(a.param);
  const float* g = reinterpret_cast<const float*>(a.grad);
  float* m = reinterpret_cast<float*>(a.exp_avg);
  float* v = reinterpret_cast<float*>(a.exp_avg_sq);
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.numel; i += stride) {
    float pi = p[i], mi = m[i], vi = v[i];
    adam_one(pi, g[i], mi, vi, a);
    p[i] = pi;
    m[i] = mi;
    v[i] = vi;
  }
}

}  // namespace

cudaError_t launch_adamw(const AdamArgs& a, cudaStream_t stream) {
  if (a.numel == 0) return cudaSuccess;
  if (a.is_bf16) {
    const size_t blocks = ((a.numel + 7) / 8 + 255) / 256;
    if (blocks > 0x7fffffffu) return cudaErrorInvalidValue;
    adamw_bf16_kernel<<<(unsigned)blocks, 256, 0, stream>>>(a);
    return cudaGetLastError();
  }
  size_t blocks = (a.numel + 255) / 256;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    sms = 132;
  if (blocks > (size_t)sms * 16) blocks = (size_t)sms * 16;
  adamw_f32_kernel<<<(unsigned)blocks, 256, 0, stream>>>(a);
  return cudaGetLastError();
}

}  // namespace epb
