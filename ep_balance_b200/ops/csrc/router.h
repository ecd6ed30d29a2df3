// Fused top-k routing for inference (router.cu): the fp32 weight split into bf16 terms, and one warp per token that turns a row
// of logits into the selected expert ids and their gate weights.  Replaces chains of PyTorch kernels (split: ~9 launches;
// sigmoid / topk / scatter / where / topk / normalise: ~15) that dominate a small-batch forward.
// Forward only: training keeps the differentiable PyTorch formulation.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace epb {

enum RouterMode : int {
  kRouterSoftmaxTopk = 0,   // top-k of the logits, softmax over the selected logits
  kRouterSigmoidTopk = 1,   // top-k of the logits, sigmoid of each selected logit
  kRouterGroupLimited = 2,  // DeepSeek-V3: sigmoid scores, groups ranked by the sum of their two best scores,
                            // top-k among the experts of the best `topk_groups` groups, weights normalised
};

// w fp32 [E, H] -> bf16 [3 E, H]: three row blocks that sum to w to 24 mantissa bits.
cudaError_t launch_router_split(const float* w, int64_t numel, void* stacked, cudaStream_t stream);

// logits fp32 [N, parts * E]: the logits of a row are the sum of its `parts` (1 or 3) blocks of E (E <= 1024,
// E % n_groups == 0), optional bias fp32 [E] added.  idx int64 [N, K], weights fp32 [N, K]; K <= 32.
cudaError_t launch_router_topk(const float* logits, const float* bias, int N, int E, int K, int mode, int n_groups,
                               int topk_groups, float scale, int64_t* idx, float* weights, cudaStream_t stream, int parts = 1);
// The three terms of the transposed matrix: w fp32 [rows, cols] -> stacked bf16 [3 cols, rows].
cudaError_t launch_router_split_transposed(const float* w, int rows, int cols, void* stacked, cudaStream_t stream);

}  // namespace epb
