// Host-side entry points of the kernel layer: launchers and the variant picker.
#pragma once
#include <cuda_runtime.h>

#include "../core/status.h"
#include "coll_args.h"

namespace amem {

// Launches one rank's kernel on `stream`.
Status launch_collective(const CollArgs& a, const LaunchPlan& plan, cudaStream_t stream);
// The same for a communicator of one rank, where that is a copy or a scale and cast of aligned buffers and
// takes no more blocks than block_cap (0: any number); *handled is false where launch_collective has to do it.
Status launch_local(const CollArgs& a, int block_cap, cudaStream_t stream, bool* handled);
// The blocks launch_local runs for this operation; 0: it does not take it.
size_t local_blocks(const CollArgs& a, int block_cap);
// dst[i][0 .. n[i]) += scale * src[i][0 .. n[i]) (fp32 += bf16) for every piece of memory i; a launch per kSumPieces pieces that are
// not empty, none of more blocks than block_cap (0: any number).
constexpr int kSumPieces = 32;
Status launch_sum_pieces(const void* const* src, float* const* dst, const long long* n, int pieces, float scale, int block_cap, cudaStream_t stream);
// The blocks that each of these launches runs, the largest of them.
size_t sum_pieces_blocks(const long long* n, int pieces, int block_cap);
// Launches every rank of an emulated (single-GPU) communicator as one cooperative grid.
// `dev_all` points to `nranks` CollArgs in device-readable memory; `a` is any rank's copy
// (used for type dispatch only).
// One thread waits, the way every collective kernel waits for a peer, until *flag >= want or
// timeout_ns have passed; a wait that runs out is recorded in `status` (host-visible words) like a
// collective's and the kernel returns normally.
Status launch_wait_probe(const uint32_t* flag, uint32_t want, unsigned long long timeout_ns, uint32_t* status, cudaStream_t stream);
Status launch_collective_emu(const CollArgs* dev_all, const CollArgs& a, int nranks, const LaunchPlan& plan, cudaStream_t stream);
int sendrecv_blocks(const CollArgs& a);

struct TunerInput {
  int kind;
  size_t count;       // elements, with the per-kind meaning of CollArgs::count
  int dtype, redop;
  int nranks;
  size_t stage_bytes, p2p_slot_bytes;
  bool nvls;          // multicast mapping available
  int max_blocks;     // upper bound for this communicator (emulated comms use a small one)
  int block_cap = 0;  // the same where the user set it (maxCTAs, AMEM_MAX_BLOCKS), 0: nobody did
  int forced_algo;    // kAlgoAuto or a variant forced by AMEM_ALGO / the API
  bool window = false;      // all-reduce: both operands lie in registered windows at vector-aligned offsets
  bool window_mc = false;   // ... and the windows have multicast mappings
};

// Deterministic in its inputs: every rank, and the same rank before and after a pause,
// gets the same variant, grid and chunking, which keeps results bitwise reproducible.
LaunchPlan plan_collective(const TunerInput& in);

}  // namespace amem
