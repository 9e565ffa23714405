// Collectives of a communicator of one rank: a copy, or a scale and cast, of the operand.  The general
// kernel runs 128 blocks with two loads in flight per thread and keeps protocol state; here every block
// moves one piece of 16 KB (copy) or 8192 elements (cast), all its loads ahead of its stores, and nothing
// else.  100 MB copied: 53 us (3.8 TB/s) before, 31.7 (6.3 TB/s) so, 35.2 with eight blocks an SM that
// stride over the buffer; bf16 to fp32, the same 50 M elements: 69 us before, 47.0 (6.4 TB/s) so.
#include <algorithm>

#include "coll_device.cuh"
#include "launch.h"
#include "pdl.cuh"

namespace amem {
namespace localk {

constexpr int THREADS = 256, AHEAD = 4, CAST_AHEAD = 8;

__global__ void __launch_bounds__(THREADS) copy_kernel(const char* src, char* dst, size_t bytes) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t n = bytes / 16, i0 = (size_t)blockIdx.x * THREADS * AHEAD + threadIdx.x;
  uint4 v[AHEAD];
#pragma unroll
  for (int j = 0; j < AHEAD; ++j)
    if (i0 + j * THREADS < n) v[j] = ((const uint4*)src)[i0 + j * THREADS];
#pragma unroll
  for (int j = 0; j < AHEAD; ++j)
    if (i0 + j * THREADS < n) ((uint4*)dst)[i0 + j * THREADS] = v[j];
  if (blockIdx.x == 0 && threadIdx.x < bytes % 16) dst[n * 16 + threadIdx.x] = src[n * 16 + threadIdx.x];
}

template <typename T>
struct alignas(4 * sizeof(T)) Four {
  T e[4];
};

// out = (TO)(scale * in), in fp32; four elements per access, so that a warp covers whole lines on both sides
template <typename TI, typename TO>
__global__ void __launch_bounds__(THREADS) scale_kernel(const TI* src, TO* dst, size_t count, float scale) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t n = count / 4, i0 = (size_t)blockIdx.x * THREADS * CAST_AHEAD + threadIdx.x;
  Four<TI> v[CAST_AHEAD];
#pragma unroll
  for (int j = 0; j < CAST_AHEAD; ++j)
    if (i0 + j * THREADS < n) v[j] = ((const Four<TI>*)src)[i0 + j * THREADS];
#pragma unroll
  for (int j = 0; j < CAST_AHEAD; ++j)
    if (i0 + j * THREADS < n) {
      Four<TO> o;
#pragma unroll
      for (int q = 0; q < 4; ++q) o.e[q] = dev::from_acc<TO, float>(dev::to_acc<TI>(v[j].e[q]) * scale);
      ((Four<TO>*)dst)[i0 + j * THREADS] = o;
    }
  if (blockIdx.x == 0 && threadIdx.x < count % 4) dst[n * 4 + threadIdx.x] = dev::from_acc<TO, float>(dev::to_acc<TI>(src[n * 4 + threadIdx.x]) * scale);
}

// dst += scale * src over several pieces of memory: the sum over one rank's gradients, tensor by tensor, added to its
// shard where the tensors lie.  A block per 4096 elements, all its loads ahead of its stores; where the user bounds the blocks, each
// takes several.  67 M elements: 107 us, of which 102 are the bytes (ten an element; through a flat buffer, a reduce-scatter
// and an add it was 26 and five passes).
constexpr int SUM_AHEAD = 2;      // vectors of eight elements a thread
constexpr size_t SUM_BLOCK = THREADS * SUM_AHEAD * 8;
struct SumPiece {
  const __nv_bfloat16* src;
  float* dst;
  size_t n;
  long first_block;
};
struct SumPieces {
  SumPiece piece[kSumPieces];
  int count;
  float scale;
  long blocks;
};
__global__ void __launch_bounds__(THREADS) sum_kernel(const __grid_constant__ SumPieces a) {
  pdl_launch_dependents();
  pdl_wait();
  int p = 0;
  for (long block = blockIdx.x; block < a.blocks; block += gridDim.x) {
    while (p + 1 < a.count && block >= a.piece[p + 1].first_block) ++p;
    const SumPiece& piece = a.piece[p];
    const __nv_bfloat16* src = piece.src;
    float* dst = piece.dst;
    const size_t base = (size_t)(block - piece.first_block) * SUM_BLOCK, n = piece.n;
    if ((((uintptr_t)src | (uintptr_t)dst) & 15) || base + SUM_BLOCK > n) {   // the end of a piece, or one at an odd place
      for (size_t i = base + threadIdx.x; i < min(n, base + SUM_BLOCK); i += THREADS) dst[i] += a.scale * __bfloat162float(src[i]);
      continue;
    }
    uint4 v[SUM_AHEAD];
    float4 d[SUM_AHEAD][2];
#pragma unroll
    for (int j = 0; j < SUM_AHEAD; ++j) {
      const size_t i = base + ((size_t)j * THREADS + threadIdx.x) * 8;
      v[j] = *(const uint4*)(src + i);
      d[j][0] = *(const float4*)(dst + i);
      d[j][1] = *(const float4*)(dst + i + 4);
    }
#pragma unroll
    for (int j = 0; j < SUM_AHEAD; ++j) {
      const size_t i = base + ((size_t)j * THREADS + threadIdx.x) * 8;
      const __nv_bfloat162* h = (const __nv_bfloat162*)&v[j];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float2 x = __bfloat1622float2(h[2 * q]), y = __bfloat1622float2(h[2 * q + 1]);
        d[j][q].x += a.scale * x.x;
        d[j][q].y += a.scale * x.y;
        d[j][q].z += a.scale * y.x;
        d[j][q].w += a.scale * y.y;
        *(float4*)(dst + i + 4 * q) = d[j][q];
      }
    }
  }
}

template <typename TI, typename TO>
cudaError_t scaled(const CollArgs& a, int grid, cudaStream_t stream) {
  return launch_overlapped(scale_kernel<TI, TO>, dim3(grid), dim3(THREADS), 0, stream, (const TI*)a.send, (TO*)a.recv, (size_t)a.count, a.scale);
}
template <typename TI>
cudaError_t scaled_from(const CollArgs& a, int grid, cudaStream_t stream) {
  return a.out_dtype == kF32 ? scaled<TI, float>(a, grid, stream) : a.out_dtype == kBF16 ? scaled<TI, __nv_bfloat16>(a, grid, stream)
                                                                                           : scaled<TI, __half>(a, grid, stream);
}

bool narrow_float(int t) { return t == kF32 || t == kBF16 || t == kF16; }

}  // namespace localk

// What a one-rank collective is as a single pass over aligned buffers: 1 a plain copy, 2 a scale and cast
// among fp32 / bf16 / fp16, 0 neither (other types with a scale, odd addresses): the general kernel's.
static int local_form(const CollArgs& a) {
  using namespace localk;
  if (a.nranks != 1 || (((uintptr_t)a.send | (uintptr_t)a.recv) & 15)) return 0;
  if (a.dtype > kBF16 || a.out_dtype > kBF16) return 0;   // 8-bit floats as such: reductions of them are refused there
  if (a.dtype == a.out_dtype && (!a.has_scale || (a.scale == 1.0f && narrow_float(a.dtype)))) return 1;
  const bool pair = a.dtype == a.out_dtype || a.dtype == kF32 || a.out_dtype == kF32;   // bf16 <-> fp16 is refused
  return narrow_float(a.dtype) && narrow_float(a.out_dtype) && pair && a.send != a.recv ? 2 : 0;
}

// A block per piece.  Where the user bounds the blocks of a communicator (maxCTAs, AMEM_MAX_BLOCKS), because
// the other SMs are for something else, what needs more of them is left to the general kernel, which strides.
size_t local_blocks(const CollArgs& a, int block_cap) {
  using namespace localk;
  const int form = local_form(a);
  if (!form) return 0;
  const size_t items = form == 1 ? a.count * dtype_size(a.dtype) / 16 : a.count / 4, per_block = (size_t)THREADS * (form == 1 ? AHEAD : CAST_AHEAD);
  const size_t blocks = std::max<size_t>(1, (items + per_block - 1) / per_block);
  return block_cap > 0 && blocks > (size_t)block_cap ? 0 : blocks;
}

// Walks the launches: f(pieces of one of them, its blocks).
template <typename F>
static Status sum_launches(const void* const* src, float* const* dst, const long long* n, int pieces, int block_cap, F&& f) {
  using namespace localk;
  SumPieces a;
  a.count = 0;
  a.blocks = 0;
  for (int i = 0; i < pieces; ++i) {
    if (n[i] > 0) {
      a.piece[a.count++] = {src ? (const __nv_bfloat16*)src[i] : nullptr, dst ? dst[i] : nullptr, (size_t)n[i], a.blocks};
      a.blocks += (long)(((size_t)n[i] + SUM_BLOCK - 1) / SUM_BLOCK);
    }
    if (a.count == kSumPieces || (i == pieces - 1 && a.count > 0)) {
      AMEM_TRY(f(a, std::min(a.blocks, block_cap > 0 ? (long)block_cap : 0x7fffffffL)));
      a.count = 0;
      a.blocks = 0;
    }
  }
  return kSuccess;
}

Status launch_sum_pieces(const void* const* src, float* const* dst, const long long* n, int pieces, float scale, int block_cap, cudaStream_t stream) {
  return sum_launches(src, dst, n, pieces, block_cap, [&](localk::SumPieces& a, long blocks) {
    a.scale = scale;
    cudaError_t e = launch_overlapped(localk::sum_kernel, dim3((unsigned)blocks), dim3(localk::THREADS), 0, stream, a);
    return e == cudaSuccess ? kSuccess : fail(kCudaError, "sum of gradients: launch failed: %s", cudaGetErrorString(e));
  });
}

size_t sum_pieces_blocks(const long long* n, int pieces, int block_cap) {
  long most = 0;
  sum_launches(nullptr, nullptr, n, pieces, block_cap, [&](localk::SumPieces&, long blocks) {
    most = std::max(most, blocks);
    return kSuccess;
  });
  return (size_t)most;
}

Status launch_local(const CollArgs& a, int block_cap, cudaStream_t stream, bool* handled) {
  using namespace localk;
  const size_t blocks = local_blocks(a, block_cap);
  const bool copy = local_form(a) == 1;
  *handled = blocks > 0;
  if (blocks == 0 || a.send == a.recv) return kSuccess;   // (in place: nothing to move)
  if (blocks > 0x7fffffffu) return fail(kInvalidArgument, "one-rank collective of %zu elements", (size_t)a.count);
  const int grid = (int)blocks;
  cudaError_t e;
  CollArgs s = a;
  if (!s.has_scale) s.scale = 1.0f;
  if (copy) e = launch_overlapped(copy_kernel, dim3(grid), dim3(THREADS), 0, stream, (const char*)a.send, (char*)a.recv, a.count * dtype_size(a.dtype));
  else if (a.dtype == kF32) e = scaled_from<float>(s, grid, stream);
  else if (a.dtype == kBF16) e = scaled_from<__nv_bfloat16>(s, grid, stream);
  else e = scaled_from<__half>(s, grid, stream);
  if (e != cudaSuccess) return fail(kCudaError, "one-rank collective launch failed: %s", cudaGetErrorString(e));
  return kSuccess;
}

}  // namespace amem
