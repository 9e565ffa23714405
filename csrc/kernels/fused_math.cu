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
#include "pdl.cuh"

namespace amem {
namespace mathk {

constexpr int THREADS = 256;
constexpr int ADAM_AHEAD = 2;   // groups of four parameters per thread: eight loads in flight
constexpr int NORM_THREADS = 512, NORM_VECS = 4;   // a row of up to 16384 elements in one block's registers

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

// Sum of v over a block of whole warps; `part` holds a value per warp and is not read again before the next
// barrier but one, so callers alternate between two of them.
__device__ __forceinline__ float block_sum(float v, float* part) {
#pragma unroll
  for (int o = 16; o > 0; o /= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x / 32, warps = blockDim.x / 32;
  if (threadIdx.x % 32 == 0) part[warp] = v;
  __syncthreads();
  float sum = 0.f;
  for (int i = 0; i < warps; ++i) sum += part[i];
  return sum;
}

// y[r] = x[r] * rstd[r] * w with rstd = 1 / sqrt(mean(x[r]^2) + eps): a block per row, which it holds in registers
// (VECS vectors of eight a thread), so x is read once.  2048 rows of 2048: 7.6 us cold under ncu, launch included, 2.6 are the
// bytes (seven torch passes: 47); the rest is the latency of one load, one reduction and one store.
template <int VECS>
__global__ void __launch_bounds__(NORM_THREADS) rms_norm_kernel(const char* x, const char* w, char* y, float* rstd, int dim, float eps) {
  __shared__ float part[NORM_THREADS / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int vecs = dim / 8;
  const long row = blockIdx.x;
  Bf8 v[VECS], wv[VECS];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c < vecs) {
      v[i] = ((const Bf8*)x)[row * vecs + c];
      wv[i] = ((const Bf8*)w)[c];
    }
  }
#pragma unroll
  for (int i = 0; i < VECS; ++i)
    if (threadIdx.x + i * blockDim.x < vecs) {
      float f[8];
      unpack(v[i], f);
#pragma unroll
      for (int q = 0; q < 8; ++q) sum = fmaf(f[q], f[q], sum);
    }
  const float r = rsqrtf(block_sum(sum, part) / (float)dim + eps);
  if (rstd && threadIdx.x == 0) rstd[row] = r;
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c < vecs) {
      float f[8], g[8];
      unpack(v[i], f);
      unpack(wv[i], g);
#pragma unroll
      for (int q = 0; q < 8; ++q) f[q] = f[q] * r * g[q];
      ((Bf8*)y)[row * vecs + c] = pack(f);
    }
  }
}

// Gradients of the above.  With n = x * rstd: g_x = rstd * (g * w - n * mean(g * w * n)), g_w = sum over rows of
// g * n.  Blocks stride over the rows and keep the columns' sums in registers; each leaves its sums in
// part_w [gridDim.x][dim] and rms_norm_weight_grad_kernel adds them in the order of the blocks.  The same size: 10.4 + 6.6 us
// (as torch passes about 130).  2048 x 8192: 46.1 us, with the next row on its way 39.9, 15 are the bytes.
template <int VECS>
__global__ void __launch_bounds__(NORM_THREADS) rms_norm_grad_kernel(const char* g_y, const char* x, const char* w, const float* rstd, char* g_x, float* part_w,
                                                                     long rows, int dim) {
  __shared__ float part[2][NORM_THREADS / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int vecs = dim / 8;
  Bf8 wv[VECS];
  float acc[VECS][8];
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c < vecs) wv[i] = ((const Bf8*)w)[c];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[i][q] = 0.f;
  }
  int flip = 0;
  // Up to two vectors a thread, the next row is on its way while this one is reduced (four leave no registers for it).
  constexpr bool AHEAD = VECS <= 2;
  Bf8 x_next[VECS], g_next[VECS];
  float r_next = 0.f;
  auto load = [&](long row, Bf8 (&xv)[VECS], Bf8 (&gv)[VECS], float& r) {
    r = rstd[row];
#pragma unroll
    for (int i = 0; i < VECS; ++i) {
      const int c = threadIdx.x + i * blockDim.x;
      if (c < vecs) {
        xv[i] = ((const Bf8*)x)[row * vecs + c];
        gv[i] = ((const Bf8*)g_y)[row * vecs + c];
      }
    }
  };
  if (AHEAD && blockIdx.x < rows) load(blockIdx.x, x_next, g_next, r_next);
  for (long row = blockIdx.x; row < rows; row += gridDim.x, flip ^= 1) {
    Bf8 xv[VECS], gv[VECS];
    float r;
    if (AHEAD) {
      r = r_next;
#pragma unroll
      for (int i = 0; i < VECS; ++i) {
        xv[i] = x_next[i];
        gv[i] = g_next[i];
      }
      if (row + gridDim.x < rows) load(row + gridDim.x, x_next, g_next, r_next);
    } else {
      load(row, xv, gv, r);
    }
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VECS; ++i)
      if (threadIdx.x + i * blockDim.x < vecs) {
        float a[8], g[8], b[8];
        unpack(xv[i], a);
        unpack(gv[i], g);
        unpack(wv[i], b);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float n = a[q] * r;
          acc[i][q] = fmaf(g[q], n, acc[i][q]);
          dot = fmaf(g[q] * b[q], n, dot);
        }
      }
    const float mean = block_sum(dot, part[flip]) / (float)dim;
    if (g_x) {
#pragma unroll
      for (int i = 0; i < VECS; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        if (c < vecs) {
          float a[8], g[8], b[8];
          unpack(xv[i], a);
          unpack(gv[i], g);
          unpack(wv[i], b);
#pragma unroll
          for (int q = 0; q < 8; ++q) a[q] = r * (g[q] * b[q] - a[q] * r * mean);
          ((Bf8*)g_x)[row * vecs + c] = pack(a);
        }
      }
    }
  }
  if (part_w) {
#pragma unroll
    for (int i = 0; i < VECS; ++i) {
      const int c = threadIdx.x + i * blockDim.x;
      if (c < vecs) {
        float4* dst = (float4*)(part_w + (size_t)blockIdx.x * dim + c * 8);
        dst[0] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        dst[1] = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
      }
    }
  }
}

// g_w[c] = sum of `blocks` partial sums: 32 columns a block, a warp per piece of the sum
__global__ void __launch_bounds__(1024) rms_norm_weight_grad_kernel(const float* part_w, __nv_bfloat16* g_w, int blocks, int dim) {
  __shared__ float sums[32][33];
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, c = blockIdx.x * 32 + lane;
  float sum = 0.f;
  if (c < dim)
    for (int b = warp; b < blocks; b += 32) sum += part_w[(size_t)b * dim + c];
  sums[warp][lane] = sum;
  __syncthreads();
  sum = sums[lane][warp];
#pragma unroll
  for (int o = 16; o > 0; o /= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0 && blockIdx.x * 32 + warp < dim) g_w[blockIdx.x * 32 + warp] = __float2bfloat16_rn(sum);
}

// (o[2i], o[2i+1]) = (x[2i], x[2i+1]) turned by the angle of (position, i), one tensor or two; a block per token, so its
// heads share the token's row of the tables out of L1.  q [1, 16, 2048, 128] and k with 4 heads: 8.3 us, 3.2 are the bytes
// (as torch passes over fp32 copies, forward and backward in the mean: 120).
__global__ void __launch_bounds__(THREADS) rotate_kernel(const __grid_constant__ Rotation a) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x / a.seq, s = blockIdx.x - b * a.seq, first = a.t[0].heads * a.vecs, all = first + a.t[1].heads * a.vecs;
  for (int i = threadIdx.x; i < all; i += blockDim.x) {
    const Rotated& t = a.t[i >= first];
    const int j = i >= first ? i - first : i, h = j / a.vecs, v = j - h * a.vecs;
    const float4 c = ((const float4*)a.cos)[(long)s * a.vecs + v], n = ((const float4*)a.sin)[(long)s * a.vecs + v];
    float x[8];
    unpack(*(const Bf8*)(t.in + (b * t.in_b + h * t.in_h + s * t.in_s) * 2 + v * 16), x);
    const float cs[4] = {c.x, c.y, c.z, c.w}, sn[4] = {n.x * a.turn, n.y * a.turn, n.z * a.turn, n.w * a.turn};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float x1 = x[2 * q], x2 = x[2 * q + 1];
      x[2 * q] = x1 * cs[q] - x2 * sn[q];
      x[2 * q + 1] = x1 * sn[q] + x2 * cs[q];
    }
    *(Bf8*)(t.out + (b * t.out_b + h * t.out_h + s * t.out_s) * 2 + v * 16) = pack(x);
  }
}

// Rows of a table's gradient (zeroed before): the first token of an id adds up the rows of all tokens that have it, in
// their order, four in flight.  A block per token; it looks through the ids 256 at a time, which is most of its work (they stay in L1: no
// shared memory to speak of), so the number of tokens is bounded by the caller.  The block of an id of `many` tokens and more would be
// busy long after the others: it marks the token and leaves the id to embedding_many_kernel.  With the zeros, L2 flushed, us (torch's
// kernel / every id its block's / so): 2048 tokens of a 32768 x 2048 table drawn evenly 146 / 32 / 34, by Zipf's law 144 / 97 / 48, all of
// one id 189 / 833 / 46; 16384 of 65536 x 4096 evenly 1397 / 204 / 191, by Zipf's law 1016 / 1285 / 249, half of them one id
// 1097 / 6458 / 239, all of them 754 / 12983 / 249, each id 70 times 759 / 235 / 155.
constexpr int MOST = 128, AHEAD = 4;   // of `many`; rows in flight
__global__ void __launch_bounds__(THREADS, 6) embedding_grad_kernel(const char* g, const long long* ids, char* g_table, unsigned char* marks, int many, int tokens, int vecs,
                                                                 long long rows) {
  __shared__ int found[MOST];
  __shared__ int before[THREADS / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const long long id = ids[t];
  if (threadIdx.x == 0) marks[t] = 0;
  if (id < 0 || id >= rows) return;
  int earlier = 0, later = 0;
  for (int i = threadIdx.x; i < t; i += THREADS) earlier |= ids[i] == id;
  if (__syncthreads_or(earlier)) return;
  for (int i = t + 1 + threadIdx.x; i < tokens; i += THREADS) later += ids[i] == id;
  if (!__syncthreads_or(later)) {   // the id's only token (its sum is the row)
    for (int v = threadIdx.x; v < vecs; v += THREADS) {
      float f[8];
      unpack(((const Bf8*)g)[(long)t * vecs + v], f);
#pragma unroll
      for (int q = 0; q < 8; ++q) f[q] += 0.f;   // (as a sum that starts at zero: no negative zeros)
      ((Bf8*)g_table)[id * vecs + v] = pack(f);
    }
    return;
  }
  later = __reduce_add_sync(0xffffffffu, later);
  if (lane == 0) before[warp] = later;
  __syncthreads();
  int all = 1;
  for (int w = 0; w < THREADS / 32; ++w) all += before[w];
  if (all >= many) {
    if (threadIdx.x == 0) marks[t] = 1;
    return;
  }
  for (int base = t, have = 0; have < all && base < tokens; base += THREADS) {
    const int i = base + threadIdx.x;
    const bool same = i < tokens && ids[i] == id;
    if (!__syncthreads_or(same)) continue;
    const unsigned mask = __ballot_sync(0xffffffffu, same);
    if (lane == 0) before[warp] = __popc(mask);
    __syncthreads();
    int at = have;
    for (int w = 0; w < THREADS / 32; ++w) {
      if (w < warp) at += before[w];
      have += before[w];
    }
    if (same) found[at + __popc(mask & ((1u << lane) - 1u))] = i;
    __syncthreads();
  }
  for (int v = threadIdx.x; v < vecs; v += THREADS) {
    float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j = 0; j < all; j += AHEAD) {
      Bf8 x[AHEAD];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u)
        if (j + u < all) x[u] = ((const Bf8*)g)[(long)found[j + u] * vecs + v];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u)
        if (j + u < all) {
          float f[8];
          unpack(x[u], f);
#pragma unroll
          for (int q = 0; q < 8; ++q) sum[q] += f[q];
        }
    }
    ((Bf8*)g_table)[id * vecs + v] = pack(sum);
  }
}

// The ids that the kernel above left a mark for.  A block takes consecutive items of (id, slice of its columns): it finds the id's tokens
// once, and GROUPS groups of threads add a part of the rows each, whose sums are added in the order of the groups.
constexpr int LOOK = 8;                              // ids a thread looks at in one go
constexpr int FOUND = 2 * LOOK * THREADS;            // positions that a block keeps
constexpr int SLICE = 8, GROUPS = THREADS / SLICE;   // vectors of a slice (a line of 128 bytes), groups of threads over its rows
constexpr int MARKS = 64 * THREADS;                  // marks that a block looks at in one go
constexpr int MANY_BLOCKS = 2 * 148;

struct Positions {
  int found[FOUND];
  int counts[LOOK][THREADS / 32];
};
// Appends the tokens i >= at that have `id`, in order, to p->found[0, have) until the ids are through or the next go might not fit; all
// threads of the block.  Moves `at` on; returns the new number.
__device__ __forceinline__ int find_tokens(const long long* ids, int tokens, long long id, int& at, int have, Positions* p) {
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  while (at < tokens && have + LOOK * THREADS <= FOUND) {
    unsigned same[LOOK];
#pragma unroll
    for (int j = 0; j < LOOK; ++j) {
      const int i = at + j * THREADS + threadIdx.x;
      same[j] = i < tokens && ids[i] == id;
    }
#pragma unroll
    for (int j = 0; j < LOOK; ++j) {
      same[j] = __ballot_sync(0xffffffffu, same[j]);
      if (lane == 0) p->counts[j][warp] = __popc(same[j]);
    }
    __syncthreads();
    int before = have;
#pragma unroll
    for (int j = 0; j < LOOK; ++j)
#pragma unroll
      for (int w = 0; w < THREADS / 32; ++w) {
        if (w == warp && (same[j] >> lane & 1u)) p->found[before + __popc(same[j] & ((1u << lane) - 1u))] = at + j * THREADS + threadIdx.x;
        before += p->counts[j][w];
      }
    have = before;
    at += LOOK * THREADS;
    __syncthreads();
  }
  return have;
}

// sum += the rows rows[from], rows[from + step], ... of g, eight of them in flight, added in this order
__device__ __forceinline__ void add_rows(const char* g, int vecs, int v, const int* rows, int from, int step, int n, float (&sum)[8]) {
  for (int j0 = from; j0 < n; j0 += 8 * step) {
    Bf8 x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (j0 + u * step < n) x[u] = ((const Bf8*)g)[(long)rows[j0 + u * step] * vecs + v];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (j0 + u * step < n) {
        float f[8];
        unpack(x[u], f);
#pragma unroll
        for (int q = 0; q < 8; ++q) sum[q] += f[q];
      }
  }
}

__global__ void __launch_bounds__(THREADS, 2) embedding_many_kernel(const char* g, const long long* ids, char* g_table, const unsigned char* marks, int tokens,
                                                                    int vecs) {
  __shared__ Positions pos;
  __shared__ int first[LOOK * THREADS], counts[THREADS / 32];
  __shared__ float sums[THREADS / 32][SLICE][8];
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, group = threadIdx.x / SLICE, sv = threadIdx.x % SLICE, slices = (vecs + SLICE - 1) / SLICE;
  long turn = blockIdx.x;   // the next items go to the blocks behind those that took the last ones
  for (long base = 0; base < tokens; base += LOOK * THREADS) {
    if (base % MARKS == 0) {   // mostly there are none
      uint4 m[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long i = base + (j * THREADS + threadIdx.x) * 16;
        m[j] = i < tokens ? ((const uint4*)marks)[i / 16] : make_uint4(0, 0, 0, 0);   // (their memory is whole vectors)
      }
      unsigned any = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) any |= m[j].x | m[j].y | m[j].z | m[j].w;
      if (!__syncthreads_or((int)any)) {
        if (tokens - base <= MARKS) return;
        base += MARKS - LOOK * THREADS;
        continue;
      }
    }
    // the marked tokens among the next LOOK * THREADS, in order
    int mine = 0;
    const long at0 = base + threadIdx.x * LOOK;
#pragma unroll
    for (int j = 0; j < LOOK; ++j) mine += at0 + j < tokens && marks[at0 + j] == 1;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += x;
    }
    if (lane == 31) counts[warp] = upto;
    __syncthreads();
    int at = upto - mine, marked = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
      if (w < warp) at += counts[w];
      marked += counts[w];
    }
#pragma unroll
    for (int j = 0; j < LOOK; ++j)
      if (at0 + j < tokens && marks[at0 + j] == 1) first[at++] = (int)(at0 + j);
    __syncthreads();
    const long items = (long)marked * slices, per = (items + gridDim.x - 1) / gridDim.x;
    int which = -1, have = 0;
    bool whole = false;       // found[0, have) are all tokens of the id
    long long id = 0;
    for (long item = turn * per; item < min(items, (turn + 1) * per); ++item) {
      const int w = (int)(item / slices), v = (int)(item - (long)w * slices) * SLICE + sv;
      if (w != which) {
        which = w;
        id = ids[first[w]];
        whole = false;
      }
      float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (whole) {
        if (v < vecs) add_rows(g, vecs, v, pos.found, group, GROUPS, have, sum);
      } else {
        int next = first[w], done = 0;
        do {
          have = find_tokens(ids, tokens, id, next, 0, &pos);
          // token number `done` + j of the id belongs to group (done + j) % GROUPS
          if (v < vecs) add_rows(g, vecs, v, pos.found, (group - done % GROUPS + GROUPS) % GROUPS, GROUPS, have, sum);
          whole = done == 0 && next >= tokens;
          done += have;
          __syncthreads();
        } while (next < tokens);
      }
      // a warp's groups, then the warps in their order
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], SLICE);
        sum[q] += __shfl_xor_sync(0xffffffffu, sum[q], 2 * SLICE);
        if (lane < SLICE) sums[warp][lane][q] = sum[q];
      }
      __syncthreads();
      if (warp == 0 && lane < SLICE && v < vecs) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          sum[q] = 0.f;
          for (int x = 0; x < THREADS / 32; ++x) sum[q] += sums[x][lane][q];
        }
        ((Bf8*)g_table)[id * vecs + v] = pack(sum);
      }
      __syncthreads();
    }
    if (items) turn = (turn + gridDim.x - (items + per - 1) / per) % gridDim.x;
    __syncthreads();
  }
}

// Threads of a block for a row of `vecs` vectors, of which each takes up to `most`: 1, 2 or 4
int norm_threads(int vecs, int most) {
  int x = 32;
  while (x < NORM_THREADS && x * most < vecs) x *= 2;
  return x;
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

Status launched(cudaError_t e, const char* what) {
  if (e != cudaSuccess) return fail(kCudaError, "%s launch failed: %s", what, cudaGetErrorString(e));
  return kSuccess;
}

}  // namespace mathk

bool rms_norm_takes(long rows, int dim) { return rows > 0 && rows <= 0x7fffffffL && dim > 0 && dim % 8 == 0 && dim <= mathk::NORM_THREADS * mathk::NORM_VECS * 8; }

Status launch_rms_norm(const void* x, const void* w, void* y, float* rstd, long rows, int dim, float eps, cudaStream_t stream) {
  namespace k = mathk;
  // With rows for every SM several times over, a row is a matter of bandwidth and a quarter of the threads reduce it for less
  // (32768 x 4096: 143 us with a vector a thread, 111 so, 82 are the bytes); with few it is one of latency.
  const int threads = k::norm_threads(dim / 8, rows >= 8 * 148 ? k::NORM_VECS : 1), per = (dim / 8 + threads - 1) / threads;
  auto kernel = per == 1 ? k::rms_norm_kernel<1> : per == 2 ? k::rms_norm_kernel<2> : k::rms_norm_kernel<4>;
  return k::launched(launch_overlapped(kernel, dim3((unsigned)rows), dim3(threads), 0, stream, (const char*)x, (const char*)w, (char*)y, rstd, dim, eps), "rms norm");
}

// Four blocks an SM: enough rows in flight, and few enough partial sums of the weight's gradient (4.8 MB at dim 2048).
int rms_norm_grad_blocks(long rows) { return (int)std::min(rows, 4L * 148); }

Status launch_rms_norm_grad(const void* g_y, const void* x, const void* w, const float* rstd, void* g_x, float* part_w, void* g_w, long rows, int dim,
                            cudaStream_t stream) {
  namespace k = mathk;
  const int threads = k::norm_threads(dim / 8, 1), per = (dim / 8 + threads - 1) / threads, blocks = rms_norm_grad_blocks(rows);
  auto kernel = per == 1 ? k::rms_norm_grad_kernel<1> : per == 2 ? k::rms_norm_grad_kernel<2> : k::rms_norm_grad_kernel<4>;
  AMEM_TRY(k::launched(launch_overlapped(kernel, dim3(blocks), dim3(threads), 0, stream, (const char*)g_y, (const char*)x, (const char*)w, rstd, (char*)g_x,
                                         part_w, rows, dim), "rms norm gradient"));
  if (!g_w) return kSuccess;
  return k::launched(launch_overlapped(k::rms_norm_weight_grad_kernel, dim3((dim + 31) / 32), dim3(1024), 0, stream, (const float*)part_w, (__nv_bfloat16*)g_w,
                                       blocks, dim), "rms norm weight gradient");
}

Status launch_embedding_grad(const void* g, const long long* ids, void* g_table, unsigned char* marks, int tokens, int dim, long long rows, cudaStream_t stream) {
  const cudaError_t e = cudaMemsetAsync(g_table, 0, (size_t)rows * dim * 2, stream);
  if (e != cudaSuccess) return mathk::launched(e, "embedding gradient (zeros)");
  // The second kernel looks for an id's tokens again, 10 us for 16384 ids: the more there are, the later that is the shorter way.  With 32 /
  // 64 / 128, us: 128 tokens of an 8192 x 8192 table, 63 of an id, 40 / 83 / 83; 2048 of 32768 x 2048, 4 of an id, 40 / 34 / 34, and by
  // Zipf's law 52 / 48 / 58; 16384 of 65536 x 4096, 70 of an id, 279 / 267 / 155.
  const int many = tokens <= 512 ? 32 : tokens <= 4096 ? 64 : mathk::MOST;
  AMEM_TRY(mathk::launched(launch_overlapped(mathk::embedding_grad_kernel, dim3(tokens), dim3(mathk::THREADS), 0, stream, (const char*)g, ids, (char*)g_table,
                                             marks, many, tokens, dim / 8, rows), "embedding gradient"));
  if (tokens < many) return kSuccess;   // no id can have so many
  return mathk::launched(launch_overlapped(mathk::embedding_many_kernel, dim3(mathk::MANY_BLOCKS), dim3(mathk::THREADS), 0, stream, (const char*)g, ids, (char*)g_table,
                                           (const unsigned char*)marks, tokens, dim / 8), "embedding gradient (frequent ids)");
}

Status launch_rotate(const Rotation& a, int batch, cudaStream_t stream) {
  const int items = (a.t[0].heads + a.t[1].heads) * a.vecs, threads = std::min(mathk::THREADS, (items + 31) / 32 * 32);
  return mathk::launched(launch_overlapped(mathk::rotate_kernel, dim3((unsigned)batch * (unsigned)a.seq), dim3(threads), 0, stream, a), "rotary embedding");
}

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
