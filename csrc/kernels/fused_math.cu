// Element-wise passes of the models and the optimizer, each ONE pass over memory: SwiGLU forward and
// backward, the AdamW update of a parameter shard.  AdamW is bound by HBM, SwiGLU by HBM and its arithmetic
// together: 16-byte accesses, all loads of a thread ahead of its stores, a block per piece of the data (fewer
// blocks that stride over it are slower, see local_coll.cu).  Arithmetic is fp32; results are rounded once,
// where they are stored.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../core/log.h"
#include "fused_math.h"

namespace amem {
namespace mathk {

constexpr int THREADS = 256;
constexpr int ADAM_AHEAD = 2;   // groups of four parameters per thread: eight loads in flight

struct alignas(16) Bf8 {
  __nv_bfloat162 h[4];
};
__device__ __forceinline__ void unpack(const Bf8& b, float (&f)[8]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 t = __bfloat1622float2(b.h[q]);
    f[2 * q] = t.x;
    f[2 * q + 1] = t.y;
  }
}
__device__ __forceinline__ Bf8 pack(const float (&f)[8]) {
  Bf8 b;
#pragma unroll
  for (int q = 0; q < 4; ++q) b.h[q] = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
  return b;
}
// 1 + exp(-x): the accurate exponential, and its quotients below rounded to the last bit (the approximate pair lost
// two to six bits of them and everything below -87.3).
__device__ __forceinline__ float one_plus_exp(float x) { return 1.f + expf(-x); }

// Threads of a block: x along a row, y over rows, one 16-byte vector each (two or four rows a thread need
// more registers than the resident warps leave: 99 us instead of 70 for the case below).
//
// act[r, c] = silu(gate[r, c]) * up[r, c]; gate and up have rows ld elements apart (the halves of one
// tensor, or two tensors).  4096 x 2 x 14336: five torch passes 409 us, this one 77.8 (4.5 TB/s; L2 flushed,
// launch included).  The bytes alone take 54; the rest is the arithmetic (61.4 with the approximate
// exponential and quotient, which are no substitute for fp32).
__global__ void __launch_bounds__(THREADS) swiglu_kernel(const char* __restrict__ gate, const char* __restrict__ up, long ld, char* __restrict__ act, long rows,
                                                          int F) {
  const int vecs = F / 8, c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= vecs) return;
  for (long r = (long)blockIdx.y * blockDim.y + threadIdx.y; r < rows; r += (long)gridDim.y * blockDim.y) {
    float g[8], u[8];
    unpack(((const Bf8*)(gate + r * ld * 2))[c], g);
    unpack(((const Bf8*)(up + r * ld * 2))[c], u);
#pragma unroll
    for (int q = 0; q < 8; ++q) g[q] = g[q] / one_plus_exp(g[q]) * u[q];
    ((Bf8*)act)[r * vecs + c] = pack(g);
  }
}

// d gate = g * up * s * (1 + gate * (1 - s)), d up = g * (gate * s), s = sigmoid(gate).  The same size, measured the
// same way through autograd: 130 us (110 with the approximate pair).
__global__ void __launch_bounds__(THREADS) swiglu_grad_kernel(const char* __restrict__ gate, const char* __restrict__ up, long ld, const char* __restrict__ g_act,
                                                               char* __restrict__ g_gate, char* __restrict__ g_up, long rows, int F) {
  const int vecs = F / 8, c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= vecs) return;
  for (long r = (long)blockIdx.y * blockDim.y + threadIdx.y; r < rows; r += (long)gridDim.y * blockDim.y) {
    float a[8], u[8], g[8], da[8], du[8];
    unpack(((const Bf8*)(gate + r * ld * 2))[c], a);
    unpack(((const Bf8*)(up + r * ld * 2))[c], u);
    unpack(((const Bf8*)g_act)[r * vecs + c], g);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float e = one_plus_exp(a[q]), s = 1.f / e;
      du[q] = g[q] * (a[q] / e);
      da[q] = g[q] * u[q] * s * (1.f + a[q] * (1.f - s));
    }
    ((Bf8*)(g_gate + r * ld * 2))[c] = pack(da);
    ((Bf8*)(g_up + r * ld * 2))[c] = pack(du);
  }
}

// One AdamW step on a shard: fp32 gradient, moments and master weights, bf16 copy of the weights.
// Reads 16 and writes 14 bytes per parameter, once (as separate torch passes: about 90; 243 M parameters
// 4.3 ms then, 1195 us so, 1115 are the bytes).
__global__ void __launch_bounds__(THREADS) adamw_kernel(const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v, float* __restrict__ w,
                                                         __nv_bfloat16* __restrict__ w16, long n, AdamW a) {
  auto one = [&](float gg, float& mm, float& vv, float& ww) {
    mm = mm * a.b1 + a.one_minus_b1 * gg;
    vv = vv * a.b2 + a.one_minus_b2 * gg * gg;
    ww = ww * a.decay - a.lr * ((mm / a.c1) / (sqrtf(vv / a.c2) + a.eps));
  };
  const long n4 = n / 4, i0 = (long)blockIdx.x * THREADS * ADAM_AHEAD + threadIdx.x;
  float4 gg[ADAM_AHEAD], mm[ADAM_AHEAD], vv[ADAM_AHEAD], ww[ADAM_AHEAD];
#pragma unroll
  for (int j = 0; j < ADAM_AHEAD; ++j) {
    const long i = i0 + j * THREADS;
    if (i < n4) {
      gg[j] = ((const float4*)g)[i];
      mm[j] = ((const float4*)m)[i];
      vv[j] = ((const float4*)v)[i];
      ww[j] = ((const float4*)w)[i];
    }
  }
#pragma unroll
  for (int j = 0; j < ADAM_AHEAD; ++j) {
    const long i = i0 + j * THREADS;
    if (i < n4) {
      one(gg[j].x, mm[j].x, vv[j].x, ww[j].x);
      one(gg[j].y, mm[j].y, vv[j].y, ww[j].y);
      one(gg[j].z, mm[j].z, vv[j].z, ww[j].z);
      one(gg[j].w, mm[j].w, vv[j].w, ww[j].w);
      ((float4*)m)[i] = mm[j];
      ((float4*)v)[i] = vv[j];
      ((float4*)w)[i] = ww[j];
      alignas(8) __nv_bfloat162 b[2] = {__floats2bfloat162_rn(ww[j].x, ww[j].y), __floats2bfloat162_rn(ww[j].z, ww[j].w)};
      ((uint2*)w16)[i] = *(const uint2*)b;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x < n % 4) {
    const long i = n4 * 4 + threadIdx.x;
    one(g[i], m[i], v[i], w[i]);
    w16[i] = __float2bfloat16_rn(w[i]);
  }
}

// x: up to a row's vectors, y: rows, for the kernels with a thread per vector
void shape_for(long rows, int vecs, dim3* grid, dim3* block) {
  int x = 32;
  while (x < THREADS && x < vecs) x *= 2;
  *block = dim3(x, THREADS / x);
  *grid = dim3((vecs + x - 1) / x, (unsigned)std::max(1L, std::min(65535L, (rows + block->y - 1) / block->y)));
}

Status launched(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(kCudaError, "%s launch failed: %s", what, cudaGetErrorString(e));
  return kSuccess;
}

}  // namespace mathk

Status launch_swiglu(const void* gate, const void* up, long ld, void* act, long rows, int F, cudaStream_t stream) {
  dim3 grid, block;
  mathk::shape_for(rows, F / 8, &grid, &block);
  mathk::swiglu_kernel<<<grid, block, 0, stream>>>((const char*)gate, (const char*)up, ld, (char*)act, rows, F);
  return mathk::launched("swiglu");
}

Status launch_swiglu_grad(const void* gate, const void* up, long ld, const void* g_act, void* g_gate, void* g_up, long rows, int F,
                          cudaStream_t stream) {
  dim3 grid, block;
  mathk::shape_for(rows, F / 8, &grid, &block);
  mathk::swiglu_grad_kernel<<<grid, block, 0, stream>>>((const char*)gate, (const char*)up, ld, (const char*)g_act, (char*)g_gate, (char*)g_up, rows, F);
  return mathk::launched("swiglu gradient");
}

Status launch_adamw(const float* g, float* m, float* v, float* w, void* w16, long n, const AdamW& a, cudaStream_t stream) {
  const long per_block = (long)mathk::THREADS * mathk::ADAM_AHEAD, blocks = std::max(1L, (n / 4 + per_block - 1) / per_block);
  if (blocks > 0x7fffffffL) return fail(kInvalidArgument, "adamw: %ld parameters", n);
  mathk::adamw_kernel<<<(int)blocks, mathk::THREADS, 0, stream>>>(g, m, v, w, (__nv_bfloat16*)w16, n, a);
  return mathk::launched("adamw");
}

}  // namespace amem
