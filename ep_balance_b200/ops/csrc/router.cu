// One warp per token.  Element e of the row lives in lane e % 32, register slot e / 32 (up to 32 slots).
// Every selection step is a warp arg-max (value descending, index ascending on ties) followed by
// masking the winner; 2*G + topk_groups + K steps in group-limited mode.
#include "router.h"

#include <cuda_bf16.h>
#include <math_constants.h>

namespace epb {
namespace {

constexpr int kMaxSlots = 32;
constexpr unsigned kFull = 0xffffffffu;
constexpr float kTinySum = 1e-20f;  // floor of the sum that the group-limited weights are normalised by

__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + expf(-x)); }

struct Best {
  float v;
  int i;
};
__device__ __forceinline__ Best better(Best a, Best b) { return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a; }
__device__ __forceinline__ Best warp_argmax(Best x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Best y{__shfl_xor_sync(kFull, x.v, o), __shfl_xor_sync(kFull, x.i, o)};
    x = better(x, y);
  }
  return x;
}

template <int kSlots>
__global__ void __launch_bounds__(256) router_topk_kernel(const float* __restrict__ logits, const float* __restrict__ bias,
                                                         int N, int E, int K, int mode, int n_groups, int topk_groups,
                                                         float scale, int64_t* __restrict__ idx,
                                                         float* __restrict__ weights, int parts) {
  const int lane = threadIdx.x & 31;
  const int t = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  if (t >= N) return;
  const float kNone = -CUDART_INF_F;
  float s[kSlots];        // selection score of each element held by this lane (-inf: absent)
  bool nan_row = false;   // a NaN logit competes as +inf; its weight, or where weights are normalised the row's, are NaN
  auto logit = [&](int e) {
    const float* row = logits + (size_t)t * parts * E + e;
    const float v = parts == 3 ? (row[0] + row[E]) + row[2 * E] : row[0];
    return bias ? v + bias[e] : v;
  };
#pragma unroll
  for (int j = 0; j < kSlots; ++j) {
    const int e = j * 32 + lane;
    float v = kNone;
    if (e < E) {
      v = logit(e);
      if (mode == kRouterGroupLimited) v = sigmoid(v);
      if (isnan(v)) {
        nan_row = true;
        v = CUDART_INF_F;
      }
    }
    s[j] = v;
  }
  if (mode == kRouterGroupLimited) {
    const int gsize = E / n_groups;
    // score of group g = sum of its two best members; lane g keeps it
    float my_group_score = kNone;
    for (int g = 0; g < n_groups; ++g) {
      float sum = 0.f;
      int taken = -1;
      for (int pass = 0; pass < 2; ++pass) {
        Best b{kNone, 0x7fffffff};
#pragma unroll
        for (int j = 0; j < kSlots; ++j) {
          const int e = j * 32 + lane;
          if (e < E && e / gsize == g && e != taken) b = better(b, Best{s[j], e});
        }
        b = warp_argmax(b);
        if (b.v > kNone) sum += b.v;
        taken = b.i;
      }
      if (lane == (g & 31)) my_group_score = (g < 32) ? sum : my_group_score;
    }
    // keep the best topk_groups groups (n_groups <= 32)
    unsigned keep = 0u;
    for (int r = 0; r < topk_groups; ++r) {
      Best b = warp_argmax(Best{lane < n_groups ? my_group_score : kNone, lane});
      keep |= 1u << b.i;
      if (lane == b.i) my_group_score = kNone;
    }
#pragma unroll
    for (int j = 0; j < kSlots; ++j) {
      const int e = j * 32 + lane;
      // experts of dropped groups compete with score 0 (they are only chosen when fewer than K remain)
      if (e < E && !((keep >> (e / gsize)) & 1u)) s[j] = 0.f;
    }
  }
  // top-K of s
  float my_val = 0.f;   // lane r keeps the r-th winner
  int my_idx = 0;
  unsigned taken = 0u;  // bit j: this lane's element j has won (a logit of -inf stays a candidate, a winner does not)
  for (int r = 0; r < K; ++r) {
    Best b{kNone, 0x7fffffff};
#pragma unroll
    for (int j = 0; j < kSlots; ++j) {
      const int e = j * 32 + lane;
      if (e < E && !((taken >> j) & 1u)) b = better(b, Best{s[j], e});
    }
    b = warp_argmax(b);
    if ((b.i & 31) == lane) taken |= 1u << (b.i >> 5);
    if (lane == r) {
      my_val = b.v;
      my_idx = b.i;
    }
  }
  // gate weights
  float w;
  if (mode == kRouterSoftmaxTopk) {
    const float top = __shfl_sync(kFull, my_val, 0);   // winners are in descending order
    float ex = lane < K ? expf(my_val - top) : 0.f;
    float sum = ex;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
    w = ex / sum;
  } else if (mode == kRouterSigmoidTopk) {
    w = sigmoid(my_val);
  } else {
    float sum = lane < K ? my_val : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
    w = my_val / fmaxf(sum, kTinySum) * scale;
  }
  if (__any_sync(kFull, nan_row) && (mode != kRouterSigmoidTopk || (lane < K && isnan(logit(my_idx))))) w = CUDART_NAN_F;
  if (lane < K) {
    idx[(size_t)t * K + lane] = my_idx;
    weights[(size_t)t * K + lane] = w;
  }
}

// x = hi + mid + lo to 24 bits, each term bf16
__device__ __forceinline__ void split3(float x, __nv_bfloat16 (&out)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    out[i] = __float2bfloat16_rn(x);
    x -= __bfloat162float(out[i]);
  }
}

__global__ void __launch_bounds__(256) router_split_kernel(const float* __restrict__ w, int64_t numel, __nv_bfloat16* __restrict__ out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < numel; i += stride) {
    __nv_bfloat16 s[3];
    split3(w[i], s);
#pragma unroll
    for (int j = 0; j < 3; ++j) out[j * numel + i] = s[j];
  }
}

// The terms of the transposed matrix: w [rows, cols] -> out [3 cols, rows].  Tiles of 32 x 32 through shared memory, so that both
// sides are whole lines.  Takes the place of a transposing copy and seven elementwise launches in the router's backward.
__global__ void __launch_bounds__(256) router_split_transposed_kernel(const float* __restrict__ w, int rows, int cols,
                                                                      __nv_bfloat16* __restrict__ out) {
  __shared__ float tile[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = warp; i < 32; i += 8)
    if (r0 + i < rows && c0 + lane < cols) tile[i][lane] = w[(size_t)(r0 + i) * cols + c0 + lane];
  __syncthreads();
  const size_t numel = (size_t)rows * cols;
#pragma unroll
  for (int i = warp; i < 32; i += 8) {
    if (c0 + i >= cols || r0 + lane >= rows) continue;
    __nv_bfloat16 s[3];
    split3(tile[lane][i], s);
#pragma unroll
    for (int j = 0; j < 3; ++j) out[j * numel + (size_t)(c0 + i) * rows + r0 + lane] = s[j];
  }
}

}  // namespace

cudaError_t launch_router_topk(const float* logits, const float* bias, int N, int E, int K, int mode, int n_groups,
                               int topk_groups, float scale, int64_t* idx, float* weights, cudaStream_t stream, int parts) {
  if (N <= 0) return cudaSuccess;
  if (parts != 1 && parts != 3) return cudaErrorInvalidValue;
  if (E < K || E > 32 * kMaxSlots || K < 1 || K > 32) return cudaErrorInvalidValue;
  if (mode == kRouterGroupLimited && (n_groups < 1 || n_groups > 32 || E % n_groups != 0 || topk_groups < 1 || topk_groups > n_groups))
    return cudaErrorInvalidValue;
  const int blocks = (N + 7) / 8;
  const int slots = (E + 31) / 32;
#define EPB_ROUTER(S)                                                                                              \
  router_topk_kernel<S><<<blocks, 256, 0, stream>>>(logits, bias, N, E, K, mode, n_groups, topk_groups, scale, idx, \
                                                    weights, parts)
  if (slots <= 2) EPB_ROUTER(2);
  else if (slots <= 4) EPB_ROUTER(4);
  else if (slots <= 8) EPB_ROUTER(8);
  else if (slots <= 16) EPB_ROUTER(16);
  else EPB_ROUTER(32);
#undef EPB_ROUTER
  return cudaGetLastError();
}

cudaError_t launch_router_split(const float* w, int64_t numel, void* stacked, cudaStream_t stream) {
  if (numel <= 0) return cudaSuccess;
  const int64_t blocks = (numel + 255) / 256;
  router_split_kernel<<<(unsigned)(blocks < 2048 ? blocks : 2048), 256, 0, stream>>>(w, numel, reinterpret_cast<__nv_bfloat16*>(stacked));
  return cudaGetLastError();
}

cudaError_t launch_router_split_transposed(const float* w, int rows, int cols, void* stacked, cudaStream_t stream) {
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  if (rows > 65535 * 32) return cudaErrorInvalidValue;  // rows of tiles are the grid's second dimension
  router_split_transposed_kernel<<<dim3((unsigned)((cols + 31) / 32), (unsigned)((rows + 31) / 32)), 256, 0, stream>>>(
      w, rows, cols, reinterpret_cast<__nv_bfloat16*>(stacked));
  return cudaGetLastError();
}

}  // namespace epb
