// GEMM for few rows of activations, host-visible description:
//   C[rows of group e, :] = A[rows of group e, :] * W[e]^T, bf16, fp32 accumulation,
// plain (one group) or grouped.  Meant for products whose time is that of reading W once.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "../core/status.h"
#include "gemm_pair.h"   // PairEpilogue

namespace amem {

struct SkinnyProblem {
  const void* A;          // bf16 [rows, K]
  const void* W;          // bf16 [groups, N, K]
  void* C;                // bf16 [rows, N], or [rows, N / 2] with a SwiGLU epilogue
  int rows, N, K;
  const int* group_off;   // device, groups + 1 offsets; null: one group of all rows
  int groups;
  int rows_per_group;     // expected (sizes the tile only)
  int epilogue;           // PairEpilogue
  float* ws;              // partial sums, skinny_gemm_ws_bytes; null: tiles are not cut along K
  unsigned int* ctr;      // skinny_gemm_ctr_words, zero between launches
  unsigned long long timeout_ns;
  unsigned int* status;   // host-mapped status words
};

// Most rows of a group that one tile takes (more rows: more tiles over the same weights).
static const int kSkinnyMaxRows = 128;

bool skinny_gemm_takes(const SkinnyProblem& p);
Status launch_skinny_gemm(const SkinnyProblem& p, int sms, cudaStream_t stream);
int skinny_gemm_tokens(const SkinnyProblem& p);   // tokens of a tile: 16, 32, 64 or kSkinnyMaxRows
// Whether launch_skinny_gemm would cut tiles along K, given a workspace.
bool skinny_gemm_cuts(const SkinnyProblem& p, int sms);
// How launch_skinny_gemm shares out the K blocks, with a workspace or without: 0 whole tiles, 1 evenly over the SMs, 2 with a tile's owner and
// its helpers.
int skinny_gemm_schedule(const SkinnyProblem& p, int sms, bool workspace);
size_t skinny_gemm_ws_bytes(int sms);
size_t skinny_gemm_ctr_words(int sms);

}  // namespace amem
