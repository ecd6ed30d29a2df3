// Gradient of the mean token cross-entropy with respect to bf16 logits (loss.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace epb {

struct CrossEntropyGradArgs {
  const float* log_prob;     // [rows, vocab], vocab % 8 == 0, 16-byte aligned
  const int64_t* targets;    // [rows]; kIgnoreIndex rows have no gradient
  const float* weight;       // number of rows that count
  const float* grad_out;     // gradient of the loss
  void* grad;                // bf16 [rows, vocab]: (exp(log_prob) - [v == target]) * *grad_out / *weight
  int rows, vocab;
};
constexpr int64_t kIgnoreIndex = -100;
cudaError_t launch_cross_entropy_backward(const CrossEntropyGradArgs& a, cudaStream_t stream);

}  // namespace epb
