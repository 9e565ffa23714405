// Element-wise passes of the models and the optimizer (host-visible).
#pragma once
#include <cuda_runtime.h>

#include "../core/status.h"

namespace amem {

// bf16, F a multiple of 8, 16-byte aligned; gate / up and their gradients have rows ld elements apart.
Status launch_swiglu(const void* gate, const void* up, long ld, void* act, long rows, int F, cudaStream_t stream);
Status launch_swiglu_grad(const void* gate, const void* up, long ld, const void* g_act, void* g_gate, void* g_up, long rows, int F,
                          cudaStream_t stream);

struct AdamW {
  float lr, b1, one_minus_b1, b2, one_minus_b2, c1, c2, eps;   // c1, c2: 1 - b^t
  float decay;                                                 // 1 - lr * weight decay
};
// Updates m, v, w (fp32) from g (fp32) and refreshes w16 (bf16) in one pass; 16-byte aligned.
Status launch_adamw(const float* g, float* m, float* v, float* w, void* w16, long n, const AdamW& a, cudaStream_t stream);

}  // namespace amem
