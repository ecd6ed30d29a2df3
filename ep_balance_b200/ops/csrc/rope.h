// Rotary embedding of the attention input: q and k of packed [B, S, 3, heads, dim] -> [B, heads, S, dim], and the gradients of
// q, k and v back into the packed one (rope.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace epb {

struct RopeArgs {
  const void* qkv;           // forward in / backward out: bf16 [B, S, 3, heads, dim]
  void* out[3];              // forward out (q, k) / backward in (q, k, v), each bf16 [B, heads, S, dim] by its strides
  int64_t stride[3][3];      // elements between batches, heads and positions of out[i] (the last dimension is dense)
  const void* cos;           // bf16 [S, dim / 2]
  const void* sin;
  int B, S, heads, dim;      // dim % 16 == 0
};
cudaError_t launch_rope(const RopeArgs& a, cudaStream_t stream);
cudaError_t launch_rope_backward(const RopeArgs& a, void* grad_qkv, cudaStream_t stream);

}  // namespace epb
