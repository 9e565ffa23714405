// The router of a mixture-of-experts layer in one kernel: logits = x * router^T, the k largest of every token and
// their softmax.  As torch passes (product, cast, top-k, sort, softmax, cast) that was six launches: 56 us for 8192
// tokens x 4096 and 8 experts and 29 for 32 tokens, now 18.4 and 5.8 (10 are the bytes of the first; the second is the
// latency of four dependent loads and the launch).
//
// Bound by reading the tokens, so the product runs on mma.sync straight from registers: a warp holds 8 tokens a
// tile as the instruction's columns and the experts as its 16 rows, and both operands are loaded as 16-byte
// vectors along K (the order of K inside a vector is the same on both sides, which is all that a sum needs).  A
// tcgen05 tile would stage 128 rows of one operand for at most 16 that matter here.  The warps of a block cut K
// evenly and add their sums in shared memory, in the order of the warps; then a warp takes a token.
#include <cuda_bf16.h>

#include <algorithm>

#include "../core/log.h"
#include "moe.h"
#include "pdl.cuh"
#include "smem_limit.h"

namespace amem {
namespace routek {

constexpr int THREADS = 512;    // at most; few tokens get all of them, many get half
constexpr int COLS = 8, ROWS = 16, STEP = 32;   // tokens and experts of a tile, K of a 16-byte vector per lane

__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Bits of a bf16 in the order of its value, NaN last (as torch sorts them).
__device__ __forceinline__ uint32_t ordered(__nv_bfloat16 v) {
  const uint32_t b = __bfloat16_as_ushort(v);
  if ((b & 0x7fffu) > 0x7f80u) return 0xffffu;
  return b & 0x8000u ? ~b & 0xffffu : b | 0x8000u;
}
__device__ __forceinline__ float value_of(uint32_t o) {
  return __bfloat162float(__ushort_as_bfloat16((unsigned short)(o & 0x8000u ? o & 0x7fffu : ~o & 0xffffu)));
}

// MT tiles of experts, NT of tokens; AHEAD vectors of every operand row in flight.
template <int MT, int NT, int AHEAD>
__global__ void __launch_bounds__(THREADS, 1) route_kernel(const char* x, const char* router, int* idx, float* weight, int T, int d, int E, int k) {
  extern __shared__ float part[];          // [warp][expert][token + 2]; the first plane then holds [token][expert]
  constexpr int TOK = NT * COLS, LD = TOK + 2;
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, warps = blockDim.x / 32, g = lane / 4, c = lane % 4;
  const int t0 = blockIdx.x * TOK, steps = (d + STEP - 1) / STEP;
  const int s0 = (int)((long)warp * steps / warps), s1 = (int)((long)(warp + 1) * steps / warps);
  const size_t row = (size_t)d * 2;
  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[m][n][q] = 0.f;
  const uint4 none = make_uint4(0, 0, 0, 0);
  for (int s = s0; s < s1; s += AHEAD) {
    uint4 xv[AHEAD][NT], rv[AHEAD][MT][2];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int at = (s + u) * STEP + c * 8;
      const bool in = s + u < s1 && at < d;      // (d is a multiple of 8: a vector is inside or outside)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int t = t0 + n * COLS + g;
        xv[u][n] = in && t < T ? *(const uint4*)(x + t * row + (size_t)at * 2) : none;
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = m * ROWS + h * 8 + g;
          rv[u][m][h] = in && e < E ? *(const uint4*)(router + e * row + (size_t)at * 2) : none;
        }
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          const uint4 a = rv[u][m][0], b = rv[u][m][1], v = xv[u][n];
          mma_16x8x16(acc[m][n], a.x, b.x, a.y, b.y, v.x, v.y);
          mma_16x8x16(acc[m][n], a.z, b.z, a.w, b.w, v.z, v.w);
        }
  }
  const int plane = MT * ROWS * LD;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float* p = part + warp * plane + (m * ROWS + g) * LD + n * COLS + c * 2;
      *(float2*)p = make_float2(acc[m][n][0], acc[m][n][1]);
      *(float2*)(p + 8 * LD) = make_float2(acc[m][n][2], acc[m][n][3]);
    }
  __syncthreads();
  for (int i = threadIdx.x; i < E * TOK; i += blockDim.x) {
    float* p = part + (i / TOK) * LD + i % TOK;
    float sum = p[0];
    for (int w = 1; w < warps; ++w) sum += p[w * plane];
    p[0] = sum;
  }
  __syncthreads();
  // a warp per token: the largest key of (value, lowest expert first) k times
  constexpr int PER = (MT * ROWS + 31) / 32;
  for (int j = warp; j < TOK && t0 + j < T; j += warps) {
    const size_t out = (size_t)(t0 + j) * k;
    uint32_t key[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane + i * 32;
      key[i] = e < E ? ordered(__float2bfloat16_rn(part[e * LD + j])) << 16 | (0xffffu - (uint32_t)e) : 0u;   // (a key is never 0)
    }
    float first = 0.f, sum = 0.f;
    for (int q = 0; q < k; ++q) {
      uint32_t best = 0;
#pragma unroll
      for (int i = 0; i < PER; ++i) best = max(best, key[i]);
      best = __reduce_max_sync(0xffffffffu, best);
#pragma unroll
      for (int i = 0; i < PER; ++i)
        if (key[i] == best) key[i] = 0;
      const float v = value_of(best >> 16);
      if (q == 0) first = v;
      const float p = expf(v - first);
      sum += p;
      if (lane == 0) {
        idx[out + q] = (int)(0xffffu - (best & 0xffffu));
        weight[out + q] = p;
      }
    }
    __syncwarp();
    for (int q = lane; q < k; q += 32) weight[out + q] = weight[out + q] / sum;
  }
}

// The gradient of the logits, bf16 [T, E]: w_j * (g_j - <w, g>) at the chosen experts, zero elsewhere; a warp per token.
__global__ void __launch_bounds__(256) route_grad_kernel(const float* g_w, const float* weight, const int* idx, __nv_bfloat16* g_logits, int T, int E, int k) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x % 32;
  const long t = (long)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  if (t >= T) return;
  const float *g = g_w + t * k, *w = weight + t * k;
  const int* e_of = idx + t * k;
  float sum = 0.f;
  for (int j = lane; j < k; j += 32) sum = fmaf(w[j], g[j], sum);
#pragma unroll
  for (int o = 16; o > 0; o /= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  for (int e = lane; e < E; e += 32) {
    float v = 0.f;
    for (int j = 0; j < k; ++j)
      if (e_of[j] == e) v = w[j] * (g[j] - sum);
    g_logits[t * E + e] = __float2bfloat16_rn(v);
  }
}

template <int MT, int NT, int AHEAD>
Status launch(const void* x, const void* router, int* idx, float* weight, int T, int d, int E, int k, int threads, cudaStream_t stream) {
  constexpr int tokens = NT * COLS;
  const size_t smem = (size_t)(threads / 32) * MT * ROWS * (tokens + 2) * sizeof(float);
  static OncePerDevice raised;
  cudaError_t e = allow_smem(raised, route_kernel<MT, NT, AHEAD>, 96 * 1024);
  if (e != cudaSuccess) return fail(kCudaError, "cudaFuncSetAttribute(routing): %s", cudaGetErrorString(e));
  e = launch_overlapped(route_kernel<MT, NT, AHEAD>, dim3((unsigned)(((long)T + tokens - 1) / tokens)), dim3(threads), smem, stream, (const char*)x,
                                    (const char*)router, idx, weight, T, d, E, k);
  if (e != cudaSuccess) return fail(kCudaError, "routing launch failed: %s", cudaGetErrorString(e));
  return kSuccess;
}

}  // namespace routek

// Tokens of a block: 8 while that leaves SMs without a block, then 16 and, with few experts, 32, so that the experts' rows
// are read (out of L2) for more tokens at once.  A block has 16 warps while there is at most one for every SM.  Of 4096 elements, 1 /
// 1024 / 16384 tokens (us): 8 experts 8.2 / 11.3 / 45, 32 experts 11 / 13 / 57, 64 experts 14 / 16 / 86, 128 experts 27 / 26 / 198,
// 256 experts 49 / 44 / 344.  From 65 experts on a block has 8 tokens, with one vector in flight: the callers in Python
// (ops/moe.py, _route_pays) leave to a library product what that makes slower.
Status launch_moe_route(const void* x, const void* router, int* idx, float* weight, int T, int d, int E, int k, cudaStream_t stream) {
  using namespace routek;
  const int sms = 148, n = T <= COLS * sms ? 1 : T <= 4 * COLS * sms ? 2 : 4;
  const int threads = T <= n * COLS * sms ? 512 : 256;
  if (E <= 16) return n == 1 ? launch<1, 1, 4>(x, router, idx, weight, T, d, E, k, threads, stream)
                     : n == 2 ? launch<1, 2, 4>(x, router, idx, weight, T, d, E, k, threads, stream) : launch<1, 4, 2>(x, router, idx, weight, T, d, E, k, threads, stream);
  if (E <= 32) return n == 1 ? launch<2, 1, 2>(x, router, idx, weight, T, d, E, k, threads, stream)
                     : n == 2 ? launch<2, 2, 2>(x, router, idx, weight, T, d, E, k, threads, stream) : launch<2, 4, 1>(x, router, idx, weight, T, d, E, k, threads, stream);
  if (E <= 64) return n == 1 ? launch<4, 1, 1>(x, router, idx, weight, T, d, E, k, 512, stream) : launch<4, 2, 1>(x, router, idx, weight, T, d, E, k, 512, stream);
  if (E <= 128) return launch<8, 1, 1>(x, router, idx, weight, T, d, E, k, 256, stream);
  return launch<16, 1, 1>(x, router, idx, weight, T, d, E, k, 256, stream);
}

Status launch_moe_route_grad(const float* g_w, const float* weight, const int* idx, void* g_logits, int T, int E, int k, cudaStream_t stream) {
  cudaError_t e = launch_overlapped(routek::route_grad_kernel, dim3((unsigned)(((long)T + 7) / 8)), dim3(256), 0, stream, g_w, weight, idx,
                                    (__nv_bfloat16*)g_logits, T, E, k);
  if (e != cudaSuccess) return fail(kCudaError, "routing gradient launch failed: %s", cudaGetErrorString(e));
  return kSuccess;
}

}  // namespace amem
