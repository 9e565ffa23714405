// Host-visible description of the tcgen05 GEMM kernels (plain, all-gather -> GEMM,
// GEMM -> reduce-scatter).  C[M,N] = A[M,K] * B[N,K]^T, bf16 operands (both K-major, i.e. the
// layout of activations [tokens, features] and of torch Linear weights [out, in]), fp32
// accumulation in tensor memory, bf16 output.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "../core/status.h"
#include "coll_args.h"

namespace amem {

static const int kGemmBM = 128, kGemmBN = 256, kGemmBK = 64, kGemmStages = 4;
static const int kGemmThreads = 320;       // warp 0: TMA producer, warp 1: MMA issuer, warps 2-5: epilogue, warps 6-9: all-gather movers
static const int kGemmThreadsTall = 384;   // 256-row tiles: eight epilogue warps (2-9), mover warps 10-11
static const int kMaxUnits = 256;          // reduce-scatter: row blocks (of 128 rows) per rank
static const int kMaxAgUnits = 1024;       // all-gather: ready flags per source rank (a flag covers GemmParams::ag_unit_rows rows)
static const int kAgPieceBytes = 8192;     // all-gather: bytes per bulk copy of the mover

enum GemmMode : int { kGemmPlain = 0, kGemmAllGather = 1, kGemmReduceScatter = 2 };

// Flags of the fused kernels; lives in every rank's control segment right after CtrlBlock,
// so it is saved and restored by pause/resume like the rest of the protocol state.
struct FusedFlags {
  uint32_t ag_ready[kMaxRanks][kMaxAgUnits]; // written by source rank s: unit u of its shard has landed (value = epoch)
  uint32_t rs_done[kMaxRanks][kMaxUnits];    // incremented by source rank s: partial tiles of row block u delivered
  uint32_t rs_expect[kMaxRanks][kMaxUnits];  // my running total of deliveries to expect per (source, row block)
};
static_assert(sizeof(FusedFlags) <= (1u << 16) - 256, "FusedFlags must fit the room kept for it behind CtrlBlock in the control segment");

struct GemmParams {
  int M, N, K;              // problem of this rank (M = all rows, gathered or to be scattered)
  int bn;                   // tile width in columns: multiple of 32, <= kGemmBN (see gemm_pick_bn)
  int tall;                 // plain / all-gather: 1 = tiles of 256 rows (two accumulators side by side in TMEM, one B tile
                            // feeds both: a third less shared-memory fill per FLOP; the epilogue is then not overlapped)
  int mode;
  void* C;                  // plain / all-gather: bf16 [M, N] row-major, leading dimension ldc
  int ldc;
  int rows_per_rank;        // M / nranks (M when nranks == 1)
  int ag_unit_rows;         // all-gather: rows of a shard announced by one ready flag (see gemm_ag_unit_rows)
  int ag_mover;             // all-gather: how the mover warp copies: 0 = bulk async copies through shared memory
                            // (one thread), 1 = plain 16-byte loads and stores by all 32 lanes; with ag_mc set,
                            // the stores are multimem.st into the multicast mapping (one per 16 bytes for all peers)
  void* ag_mc;              // all-gather: multicast mapping of the gathered buffers (null: none)
  int ag_mover_warps;       // all-gather: mover warps per CTA that take part (1 .. 4 with 128-row tiles, 1 .. 2 with 256-row tiles)
  int ag_epi_help;          // all-gather: epilogue warps move units of the shard while they wait for an accumulator
  int copy_own;             // all-gather: also place my own shard in the gathered buffer
  const void* a_local;      // all-gather: my shard, bf16 [rows_per_rank, K]
  void* ag_buf[kMaxRanks];  // all-gather: every rank's gathered-A buffer [M, K]; [rank] is mine
  void* rs_buf[kMaxRanks];  // reduce-scatter: every rank's partial buffer, tile-major [nranks][row blocks][col blocks][128 x 256]
  void* rs_out;             // reduce-scatter: bf16 [rows_per_rank, N]
  FusedFlags* fflags[kMaxRanks];
  // Split-K of the last, partly filled wave of tiles (plain and all-gather modes): each of its tiles is cut in
  // sk_slices ranges of K that run on different CTAs; partial accumulators meet in sk_ws
  // (fp32, [tile][slice][32-column chunk][128 rows][32]) and are summed in slice order.
  int sk_slices;            // 0 or 1: off
  float* sk_ws;
  uint32_t* sk_ctr;         // two counters per tail tile (arrived, finished), zero between launches
  CollArgs coll;            // rank, nranks, control blocks, status words, timeout
};

struct GemmLaunch {
  GemmParams p;
  CUtensorMap map_a;        // plain/RS: A [M, K]; all-gather: the gathered buffer [M, K]
  CUtensorMap map_a_local;  // all-gather: my own shard [rows_per_rank, K]
  CUtensorMap map_b;        // B [N, K]
  int grid;                 // CTAs (per rank)
};

// Encodes a 2-D bf16 row-major tensor map with a [box_rows, 64] box and the 128-byte swizzle.
Status make_tensor_map_bf16(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld_elems, uint32_t box_rows);

size_t gemm_smem_bytes();
Status launch_gemm(const GemmLaunch& g, cudaStream_t stream);
// All ranks of an emulated communicator in one cooperative grid (blockIdx.y = rank).
Status launch_gemm_emu(const GemmLaunch* ranks, int nranks, cudaStream_t stream);
int gemm_default_grid(int device);
// Tile width that minimises (waves of tiles) x (tile width) for `ctas` compute CTAs.  With
// `k_blocks` > 0 the last wave may be split along K (see GemmParams::sk_slices): its cost is
// then 1/slices of a wave plus the fix-up, and *slices receives the split to use (1 = none).
int gemm_pick_bn(int row_tiles, int N, int ctas, int k_blocks = 0, int* slices = nullptr);
// Whether 256-row tiles (GemmParams::tall) are expected to beat 128-row tiles for this problem.
bool gemm_tall_pays(int M, int N, int k_blocks, int ctas, int bn_flat, int slices_flat, int bn_tall, int slices_tall);
// Slices of the tail split for a given tiling, 1 when splitting does not pay.
int gemm_tail_slices(long tiles, int ctas, int k_blocks);
// Which all-gather -> GEMM schedule a communicator of n ranks runs: mover warps inside every CTA
// (this file; the faster one up to four ranks) or dedicated mover CTAs (gemm_ag_cta_movers.cu; the
// faster one from five ranks up, where the transfer takes as long as the GEMM).
// AMEM_AG_DESIGN: 0 = by rank count, 1 = mover warps, 2 = mover CTAs.
bool gemm_ag_uses_mover_warps(int nranks);
// Rows per ready flag of the all-gather mode: as few as the flag array and the mover's copy size allow,
// so that rows become usable in the order they arrive.
int gemm_ag_unit_rows(int rows_per_rank, int K);
// Bytes of split-K workspace / number of counters that a launch on `ctas` CTAs may touch.
size_t gemm_splitk_ws_bytes(int ctas);
size_t gemm_splitk_ctr_words(int ctas);

}  // namespace amem
