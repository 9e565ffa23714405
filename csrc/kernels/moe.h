// MoE expert-parallel dispatch / combine (host-visible description).
//
// dispatch: every (token, choice) pair is written straight into the destination rank's
//           receive buffer at its final, expert-sorted row, so the routing permutation IS the
//           all-to-all: no local permute pass, no staging copy.  Row order inside an expert is
//           (source rank, token order) and is computed with scans, not atomics, so the layout
//           is identical from run to run.
// combine : the token owner pulls the k expert outputs of each token directly from the expert
//           ranks' output buffers (peer loads over NVLink), multiplies by the routing weights
//           and sums in fp32: the un-permute, the all-to-all back and the weighted sum in one
//           pass with no landing buffer.
#pragma once
#include <cuda_runtime.h>

#include "../core/status.h"
#include "coll_args.h"

namespace amem {

static const int kMoeMaxExperts = 256;   // CtrlBlock::xchg row length
static const int kMoeSegments = 148;     // CTAs of the count / scatter kernels: one per SM of a B200; any number is correct on any GPU

struct MoeArgs {
  CollArgs coll;
  int T, k, d;              // tokens on this rank, choices per token, hidden size (bf16 elements)
  int E;                    // experts over the whole communicator (E % nranks == 0)
  int capacity_rows;        // rows each rank's receive buffer can hold
  const void* x;            // bf16 [T, d]
  const int* topk_idx;      // int32 [T, k], global expert ids
  const float* topk_w;      // fp32 [T, k] (combine)
  char* recv[kMaxRanks];    // dispatch: every rank's receive buffer, bf16 [capacity_rows, d]
  char* ybuf[kMaxRanks];    // combine: every rank's expert-output buffer, bf16 [capacity_rows, d]
  void* out;                // combine: bf16 [T, d]
  // work buffers in this rank's own memory
  int* seg_hist;            // [kMoeSegments][E]
  int* seg_base;            // [kMoeSegments][E]  exclusive scan of seg_hist over segments
  int* send_off;            // [E]  first row, in the owner's buffer, of my pairs for expert e
  int* send_pos;            // [T*k] destination row of each pair (-1: dropped for capacity)
  int* expert_counts;       // [E / nranks] rows received per local expert
  int* expert_offsets;      // [E / nranks + 1] exclusive scan of expert_counts (last = total rows)
  int* dropped_rows;        // optional, one int: rows routed to this rank that did not fit capacity_rows
};

// Capacity.  A rank can be sent more rows than its buffers hold (routing is data dependent).
// That is a result of the call, not an error of the communicator: the rows that would land at
// or beyond capacity_rows are not sent (their send_pos is -1 and combine gives them weight 0),
// expert_counts / expert_offsets describe only the rows that were stored (so offsets never
// point past the buffer), and *dropped_rows says how many were left out on this rank.

Status launch_moe_dispatch(const MoeArgs& a, cudaStream_t stream);
Status launch_moe_combine(const MoeArgs& a, cudaStream_t stream);
// Whether one rank's combine gathers its rows by bulk copies.
bool moe_combine_streams(int T, int k, int d);
// Backward of the combine on one rank: g_w fp32 [T, k] and g_y bf16 [rows, d] (the rows that send_pos names;
// positions at or beyond rows count as dropped).
Status launch_moe_combine_grad(const void* g_out, const void* y, const float* w, const int* send_pos, void* g_y, float* g_w, int rows, int T, int k,
                               int d, cudaStream_t stream);
// Routing of T > 0 tokens, bf16 [T, d] with d a multiple of 8, to the k largest of their E <= kMoeMaxExperts logits (x times
// the rows of router, bf16 [E, d], rounded to bf16; equal ones by the lower expert, NaN above all), largest first:
// idx int32 and weight fp32 [T, k], the softmax over the chosen.  Its gradient down to the logits, bf16 [T, E].
Status launch_moe_route(const void* x, const void* router, int* idx, float* weight, int T, int d, int E, int k, cudaStream_t stream);
Status launch_moe_route_grad(const float* g_w, const float* weight, const int* idx, void* g_logits, int T, int E, int k, cudaStream_t stream);
// Gradient of the tokens on one rank, through the dispatch and the routing at once: g_x[t] = sum over its choices of the row's
// gradient (g_rows bf16 [rows, d] at send_pos; positions at or beyond rows count as dropped) and of the logit's gradient (g_logits
// bf16 [T, E]) times the chosen expert's row of router.
Status launch_moe_input_grad(const void* g_rows, const int* send_pos, const int* idx, const void* g_logits, const void* router, void* g_x, int rows, int T,
                             int k, int d, int E, cudaStream_t stream);
// Emulated communicator: all ranks in one cooperative grid per phase.
Status launch_moe_dispatch_emu(const MoeArgs* host_all, const MoeArgs* dev_all, int nranks, cudaStream_t stream);
Status launch_moe_combine_emu(const MoeArgs* host_all, const MoeArgs* dev_all, int nranks, cudaStream_t stream);

}  // namespace amem
