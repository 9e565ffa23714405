// Element-wise passes of the models and the optimizer (host-visible).
#pragma once
#include <cuda_runtime.h>

#include "../core/status.h"

namespace amem {

// bf16, F a multiple of 8, 16-byte aligned; gate / up and their gradients have rows ld elements apart.
Status launch_swiglu(const void* gate, const void* up, long ld, void* act, long rows, int F, cudaStream_t stream);
Status launch_swiglu_grad(const void* gate, const void* up, long ld, const void* g_act, void* g_gate, void* g_up, long rows, int F,
                          cudaStream_t stream);

// Root-mean-square norm of bf16 rows (contiguous, 16-byte aligned): y = x * rstd * w, rstd = 1 / sqrt(mean(x^2) + eps) in
// fp32, kept for the gradients where rstd is given.
bool rms_norm_takes(long rows, int dim);
Status launch_rms_norm(const void* x, const void* w, void* y, float* rstd, long rows, int dim, float eps, cudaStream_t stream);
// Its gradients; either may be null.  part_w: fp32 [rms_norm_grad_blocks(rows)][dim] of work memory for g_w.
int rms_norm_grad_blocks(long rows);
Status launch_rms_norm_grad(const void* g_y, const void* x, const void* w, const float* rstd, void* g_x, float* part_w, void* g_w, long rows, int dim,
                            cudaStream_t stream);

// g_table[rows, dim] = the sums of the rows of g[tokens, dim] over equal ids, fp32 inside, in an order that the ids alone decide; zero
// elsewhere.  Ids outside the table are left out.  marks: `tokens` bytes of work memory in whole 16-byte vectors.
Status launch_embedding_grad(const void* g, const long long* ids, void* g_table, unsigned char* marks, int tokens, int dim, long long rows,
                             cudaStream_t stream);
// Rotary embedding of bf16 [batch, heads, seq, 8 * vecs] tensors with any strides (in elements, multiples of 8) but a
// dense last dimension; cos and sin are fp32 [seq, 4 * vecs], turn = 1 or, for the gradients, -1.  The second tensor is
// left out where it has no heads.
struct Rotated {
  const char* in;
  char* out;
  int heads;
  long in_b, in_h, in_s, out_b, out_h, out_s;
};
struct Rotation {
  Rotated t[2];
  const float *cos, *sin;
  int seq, vecs;
  float turn;
};
Status launch_rotate(const Rotation& a, int batch, cudaStream_t stream);

struct AdamW {
  float lr, b1, one_minus_b1, b2, one_minus_b2, c1, c2, eps;   // c1, c2: 1 - b^t
  float decay;                                                 // 1 - lr * weight decay
};
// Updates m, v, w (fp32) from g (fp32) and refreshes w16 (bf16) in one pass; 16-byte aligned.
Status launch_adamw(const float* g, float* m, float* v, float* w, void* w16, long n, const AdamW& a, cudaStream_t stream);

}  // namespace amem
