// GEMM on pairs of SMs (tcgen05 cta_group::2), host-visible description.
//
//   C = A * B, bf16 operands, fp32 accumulation in tensor memory, bf16 result.
//
// Either operand may be stored with its contraction index contiguous (K-major: activations
// [M, K], a Linear weight [N, K]) or with its other index contiguous (A as [K, M], B as [K, N]),
// so the products of a backward pass read the tensors of the forward pass as they lie in memory.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "../core/status.h"

namespace amem {

// kPairPlain        C [M, N]
// kPairGroupedRows  rows [off[e], off[e+1]) of A [rows, K] times matrix e of B; C has A's rows
// kPairGroupedK     C [groups, M, N]: C[e] sums over rows [off[e], off[e+1]) of A [rows, M] and B [rows, N]
//                   (both with their rows as the contraction index; an empty group gives zeros)
enum PairMode : int { kPairPlain = 0, kPairGroupedRows = 1, kPairGroupedK = 2 };
// kPairStore        C as computed
// kPairSwiGLU32     B's rows alternate in blocks of 32 gate and 32 up rows; C has N / 2 columns: silu(gate) * up
// kPairSwiGLUHalves B's first N / 2 rows are the gate's, the others the up projection's; C as for kPairSwiGLU32
enum PairEpilogue : int { kPairStore = 0, kPairSwiGLU32 = 1, kPairSwiGLUHalves = 2 };

struct PairProblem {
  const void* A;
  const void* B;
  void* C;
  int a_mn, b_mn;         // 1: stored with the contraction index outermost
  int M, N, K;            // kPairGroupedRows: M = rows of A at most; kPairGroupedK: K = rows at most
  int mode, epilogue;
  const int* group_off;   // device, groups + 1 offsets
  int groups;             // 1 for kPairPlain
  int row_tiles_hint;     // grouped: row tiles of 256 expected over all groups (sizes the tile width only)
  unsigned long long timeout_ns;
  unsigned int* status;   // host-mapped status words
  // kPairPlain: workspace that lets a problem of few tiles be cut along K (null: never cut);
  // pair_gemm_ws_bytes / pair_gemm_ctr_words, counters zero between launches
  float* sk_ws;
  unsigned int* sk_ctr;
};

size_t pair_gemm_ws_bytes(int sms);
size_t pair_gemm_ctr_words(int sms);

// Whether the operands' addresses and pitches allow TMA (16-byte rule) and the sizes fit.
bool pair_gemm_takes(const PairProblem& p);
Status launch_pair_gemm(const PairProblem& p, int sms, cudaStream_t stream);
// The tiling that launch_pair_gemm takes; slices: cuts of every tile along K (1: none, and the workspace is
// not touched), more than one only where may_cut says that there is, or would be, a workspace.
struct PairTiling {
  int bn, slices;
};
PairTiling pair_gemm_tiling(const PairProblem& p, int sms, bool may_cut);
// Tile width in columns (multiple of 32, 128..256) for `row_tiles` rows of 256-row tiles on `clusters`
// SM pairs.  With `slices`, a problem that leaves half of the pairs idle may be cut along its k_blocks
// blocks of 64; *slices receives the number of cuts (1: none).
int pair_gemm_pick_bn(long row_tiles, int N, int clusters, int k_blocks, int* slices);

// Tensor map of a bf16 array [z][outer][inner] with boxes of 64 (inner) x box_outer in the 128-byte swizzle.
Status make_bf16_map(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t z, uint32_t box_outer);

}  // namespace amem
