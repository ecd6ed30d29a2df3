// Elementwise pieces of a dense block's inference forward (dense.cu), bf16 with the roundings of the operations they replace.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace epb {

// out[r, f] = round(silu(x[r, f])) * x[r, F + f]; F % 8 == 0, 16-byte aligned rows.
cudaError_t launch_swiglu(const void* x, void* out, int64_t rows, int F, cudaStream_t stream);
// out = round(a + b) + c; numel % 8 == 0.
cudaError_t launch_add3(const void* a, const void* b, const void* c, void* out, int64_t numel, cudaStream_t stream);

}  // namespace epb
