/* NCCL-compatible C API of the B200-native pausable collective library.
 *
 * Function names, argument order, enum values and the 128-byte ncclUniqueId follow NCCL 2.27 so
 * that code written against nccl.h (including ctypes loaders that look symbols up by name)
 * works unchanged.  On top of that come the five AMem entry points the reference adds to
 * nccl.h (nccl_patch/nccl_2.27.5-1.diff:329-355) -- ncclPause, ncclResume, ncclMemStats,
 * ncclSetGroupID, ncclGetGroupID -- and a small set of amem* extensions for the fused
 * operations and for observability.
 */
#ifndef AMEM_B200_NCCL_H_
#define AMEM_B200_NCCL_H_

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

#define NCCL_MAJOR 2
#define NCCL_MINOR 27
#define NCCL_PATCH 5
#define NCCL_SUFFIX "+amem.b200"
#define NCCL_VERSION_CODE 22705
#define NCCL_VERSION(X, Y, Z) (((X) <= 2 && (Y) <= 8) ? (X) * 1000 + (Y) * 100 + (Z) : (X) * 10000 + (Y) * 100 + (Z))

typedef struct CUstream_st* cudaStream_t;
typedef struct ncclComm* ncclComm_t;
typedef struct ncclWindow* ncclWindow_t;
#define NCCL_COMM_NULL NULL

#define NCCL_UNIQUE_ID_BYTES 128
typedef struct { char internal[NCCL_UNIQUE_ID_BYTES]; } ncclUniqueId;

typedef enum {
  ncclSuccess = 0,
  ncclUnhandledCudaError = 1,
  ncclSystemError = 2,
  ncclInternalError = 3,
  ncclInvalidArgument = 4,
  ncclInvalidUsage = 5,
  ncclRemoteError = 6,
  ncclInProgress = 7,
  ncclNumResults = 8
} ncclResult_t;

#define NCCL_CONFIG_UNDEF_INT INT32_MIN
#define NCCL_CONFIG_UNDEF_PTR NULL
#define NCCL_SPLIT_NOCOLOR -1

typedef struct ncclConfig_v22700 {
  size_t size;
  unsigned int magic;
  unsigned int version;
  int blocking;
  int cgaClusterSize;
  int minCTAs;
  int maxCTAs;
  const char* netName;
  int splitShare;
  int trafficClass;
  const char* commName;
  int collnetEnable;
  int CTAPolicy;
  int shrinkShare;
  int nvlsCTAs;
} ncclConfig_t;

#define NCCL_CONFIG_INITIALIZER {                                   \
  sizeof(ncclConfig_t), 0xcafebeef, NCCL_VERSION_CODE,              \
  NCCL_CONFIG_UNDEF_INT, NCCL_CONFIG_UNDEF_INT, NCCL_CONFIG_UNDEF_INT, NCCL_CONFIG_UNDEF_INT, \
  NCCL_CONFIG_UNDEF_PTR, NCCL_CONFIG_UNDEF_INT, NCCL_CONFIG_UNDEF_INT, NCCL_CONFIG_UNDEF_PTR, \
  NCCL_CONFIG_UNDEF_INT, NCCL_CONFIG_UNDEF_INT, NCCL_CONFIG_UNDEF_INT, NCCL_CONFIG_UNDEF_INT }

typedef enum { ncclSum = 0, ncclProd = 1, ncclMax = 2, ncclMin = 3, ncclAvg = 4, ncclNumOps = 5, ncclMaxRedOp = 0x7fffffff } ncclRedOp_t;

typedef enum {
  ncclInt8 = 0, ncclChar = 0,
  ncclUint8 = 1,
  ncclInt32 = 2, ncclInt = 2,
  ncclUint32 = 3,
  ncclInt64 = 4,
  ncclUint64 = 5,
  ncclFloat16 = 6, ncclHalf = 6,
  ncclFloat32 = 7, ncclFloat = 7,
  ncclFloat64 = 8, ncclDouble = 8,
  ncclBfloat16 = 9,
  ncclFloat8e4m3 = 10, /* copy collectives only: all-gather, all-to-all, broadcast, send/recv */
  ncclFloat8e5m2 = 11,
  ncclNumTypes = 12
} ncclDataType_t;

/* ---- memory ------------------------------------------------------------------------- */
/* VMM allocation on the current device, tracked by the registry and therefore pausable:
 * its contents are saved on ncclPause and restored at the same address on ncclResume. */
ncclResult_t ncclMemAlloc(void** ptr, size_t size);
ncclResult_t ncclMemFree(void* ptr);

/* ---- communicator ------------------------------------------------------------------- */
ncclResult_t ncclGetVersion(int* version);
ncclResult_t ncclGetUniqueId(ncclUniqueId* uniqueId);
ncclResult_t ncclCommInitRank(ncclComm_t* comm, int nranks, ncclUniqueId commId, int rank);
ncclResult_t ncclCommInitRankConfig(ncclComm_t* comm, int nranks, ncclUniqueId commId, int rank, ncclConfig_t* config);
ncclResult_t ncclCommInitAll(ncclComm_t* comms, int ndev, const int* devlist);
ncclResult_t ncclCommFinalize(ncclComm_t comm);
ncclResult_t ncclCommDestroy(ncclComm_t comm);
ncclResult_t ncclCommAbort(ncclComm_t comm);
ncclResult_t ncclCommSplit(ncclComm_t comm, int color, int key, ncclComm_t* newcomm, ncclConfig_t* config);
const char* ncclGetErrorString(ncclResult_t result);
const char* ncclGetLastError(ncclComm_t comm);
ncclResult_t ncclCommGetAsyncError(ncclComm_t comm, ncclResult_t* asyncError);
ncclResult_t ncclCommCount(const ncclComm_t comm, int* count);
ncclResult_t ncclCommCuDevice(const ncclComm_t comm, int* device);
ncclResult_t ncclCommUserRank(const ncclComm_t comm, int* rank);
/* Buffer registration is accepted for source compatibility; the push protocol needs none. */
ncclResult_t ncclCommRegister(const ncclComm_t comm, void* buff, size_t size, void** handle);
ncclResult_t ncclCommDeregister(const ncclComm_t comm, void* handle);
ncclResult_t ncclCommWindowRegister(ncclComm_t comm, void* buff, size_t size, ncclWindow_t* win, int winFlags);
ncclResult_t ncclCommWindowDeregister(ncclComm_t comm, ncclWindow_t win);
/* Several unique ids may be passed for source compatibility; the first one is the meeting point. */
ncclResult_t ncclCommInitRankScalable(ncclComm_t* newcomm, int nranks, int myrank, int nId, ncclUniqueId* commIds, ncclConfig_t* config);
/* Not supported (returns ncclInvalidUsage): a communicator cannot lose ranks; create a new one. */
ncclResult_t ncclCommShrink(ncclComm_t comm, int* excludeRanksList, int excludeRanksCount, ncclComm_t* newcomm, ncclConfig_t* config, int shrinkFlags);

/* Pre-multiplied sum: sum_r (scalar * x_r).  The scalar is read when the operator is created. */
typedef enum { ncclScalarDevice = 0, ncclScalarHostImmediate = 1 } ncclScalarResidence_t;
ncclResult_t ncclRedOpCreatePreMulSum(ncclRedOp_t* op, void* scalar, ncclDataType_t datatype, ncclScalarResidence_t residence, ncclComm_t comm);
ncclResult_t ncclRedOpDestroy(ncclRedOp_t op, ncclComm_t comm);

/* ---- collectives -------------------------------------------------------------------- */
ncclResult_t ncclReduce(const void* sendbuff, void* recvbuff, size_t count, ncclDataType_t datatype, ncclRedOp_t op, int root, ncclComm_t comm, cudaStream_t stream);
ncclResult_t ncclBcast(void* buff, size_t count, ncclDataType_t datatype, int root, ncclComm_t comm, cudaStream_t stream);
ncclResult_t ncclBroadcast(const void* sendbuff, void* recvbuff, size_t count, ncclDataType_t datatype, int root, ncclComm_t comm, cudaStream_t stream);
ncclResult_t ncclAllReduce(const void* sendbuff, void* recvbuff, size_t count, ncclDataType_t datatype, ncclRedOp_t op, ncclComm_t comm, cudaStream_t stream);
ncclResult_t ncclReduceScatter(const void* sendbuff, void* recvbuff, size_t recvcount, ncclDataType_t datatype, ncclRedOp_t op, ncclComm_t comm, cudaStream_t stream);
ncclResult_t ncclAllGather(const void* sendbuff, void* recvbuff, size_t sendcount, ncclDataType_t datatype, ncclComm_t comm, cudaStream_t stream);
/* count = elements exchanged with EACH peer; block j of sendbuff goes to rank j. */
ncclResult_t ncclAlltoAll(const void* sendbuff, void* recvbuff, size_t count, ncclDataType_t datatype, ncclComm_t comm, cudaStream_t stream);
ncclResult_t ncclSend(const void* sendbuff, size_t count, ncclDataType_t datatype, int peer, ncclComm_t comm, cudaStream_t stream);
ncclResult_t ncclRecv(void* recvbuff, size_t count, ncclDataType_t datatype, int peer, ncclComm_t comm, cudaStream_t stream);
ncclResult_t ncclGroupStart(void);
ncclResult_t ncclGroupEnd(void);

/* Filled by ncclGroupSimulateEnd: the group is closed without being launched and its duration
 * (microseconds) is estimated. */
typedef struct ncclSimInfo_v22200 {
  size_t size;
  unsigned int magic;
  unsigned int version;
  float estimatedTime;
} ncclSimInfo_t;
#define NCCL_UNDEF_FLOAT -1.0f
#define NCCL_SIM_INFO_INITIALIZER { sizeof(ncclSimInfo_t), 0x74685283, NCCL_VERSION_CODE, NCCL_UNDEF_FLOAT }
ncclResult_t ncclGroupSimulateEnd(ncclSimInfo_t* simInfo);
/* Re-reads the logging environment (GMM_LOG). */
void ncclResetDebugInit(void);

/* ---- AMem: pause / resume ------------------------------------------------------------ */
/* comm == NULL (or *comm == NULL): every communicator of the process plus ncclMemAlloc
 * memory.  Otherwise only that communicator.  Synchronous; every rank of the communicator
 * must call; idempotent.  After ncclPause returns, the physical memory behind the
 * communicator (this rank's and its mappings of the peers') has been returned to the driver
 * while all virtual addresses stay reserved.  Collectives issued while paused fail with
 * ncclInvalidUsage. */
ncclResult_t ncclPause(ncclComm_t* comm);
ncclResult_t ncclResume(ncclComm_t* comm);
ncclResult_t ncclMemStats(void);
/* Only before the first tracked allocation of the process; distinguishes co-located groups
 * (for instance training = 100, inference = 200). */
ncclResult_t ncclSetGroupID(int id);
ncclResult_t ncclGetGroupID(int* id);

/* ---- amem extensions ------------------------------------------------------------------ */
typedef struct {
  uint64_t bytes_by_tag[16];
  uint64_t stateful_bytes, scratch_bytes, imported_bytes, multicast_bytes;
  uint64_t live_bytes, paused_bytes, shadow_bytes;
  uint64_t n_local, n_imported;
  uint64_t pause_count, resume_count;
  int group_id;
  int paused;
} amemMemStats_t;

typedef struct {
  double quiesce_us, offload_us, release_import_us, release_local_us, pause_barrier_us, pause_total_us;
  double create_map_us, agree_us, exchange_us, import_us, preload_us, resume_barrier_us, resume_total_us;
  uint64_t bytes_offloaded, bytes_preloaded;
  uint64_t bytes_released_local, bytes_released_peer;
  uint64_t n_offload, n_release_local, n_release_peer;
  uint64_t free_before_pause, free_after_pause, free_after_resume;
} amemPauseResumeStats_t;

ncclResult_t amemMemStatsGet(amemMemStats_t* out);
/* Phase timings and byte counts of the most recent pause and resume (comm NULL: process). */
ncclResult_t amemPauseResumeStatsGet(ncclComm_t comm, amemPauseResumeStats_t* out);

/* Reduce-scatter fused with a scale and an output type cast: recv[i] = (out_type)(scale *
 * sum_r send_r[rank*recvcount + i]).  fp32 <-> bf16/fp16 and same-type are supported. */
ncclResult_t amemReduceScatterScaleCast(const void* sendbuff, void* recvbuff, size_t recvcount, ncclDataType_t in_type,
                                        ncclDataType_t out_type, float scale, ncclComm_t comm, cudaStream_t stream);
/* All-reduce with a forced variant: 1 one-shot, 2 two-shot, 3 NVLS (0 lets the tuner pick). */
ncclResult_t amemAllReduceAlgo(const void* sendbuff, void* recvbuff, size_t count, ncclDataType_t datatype, ncclRedOp_t op,
                               int algo, ncclComm_t comm, cudaStream_t stream);
/* tcgen05 GEMM, bf16 in / fp32 accumulate / bf16 out: C[M,N] = A[M,K] * B[N,K]^T (both operands
 * row-major with K contiguous, the layout of activations and of Linear weights).  N and K must
 * be multiples of 8. */
ncclResult_t amemGemmBf16(const void* A, const void* B, void* C, int M, int N, int K, cudaStream_t stream);
/* The same product with either operand stored by its contraction index: a_by_k: A is [K, M], b_by_k: B is
 * [K, N].  Built: (0, 0), (0, 1) -- a Linear's input gradient from its weight as it lies -- and (1, 1), its
 * weight gradient (K is then any number).  The contiguous extents must be multiples of 8. */
ncclResult_t amemGemmBf16Strided(const void* A, const void* B, void* C, int M, int N, int K, int a_by_k, int b_by_k, cudaStream_t stream);
/* C[M,F] = silu(A * W[0:F]^T) * (A * W[F:2F]^T), W bf16 [2 F, K]: an MLP's gate / up projection with its
 * activation in the epilogue (fp32 accumulators, one rounding). */
ncclResult_t amemGemmSwiGLU(const void* A, const void* W, void* C, int M, int F, int K, cudaStream_t stream);
/* act[r,c] = silu(gate[r,c]) * up[r,c] in bf16, and its gradients; gate, up and their gradients have rows
 * ld elements apart, act and g_act are contiguous; F and ld multiples of 8. */
ncclResult_t amemSwiGLU(const void* gate, const void* up, long long ld, void* act, long long rows, int F, cudaStream_t stream);
ncclResult_t amemSwiGLUGrad(const void* gate, const void* up, long long ld, const void* g_act, void* g_gate, void* g_up, long long rows, int F,
                            cudaStream_t stream);
/* y[r] = x[r] * rstd[r] * w, rstd[r] = 1 / sqrt(mean(x[r]^2) + eps): bf16 rows of dim elements (a multiple of 8 up to
 * 16384), fp32 inside; rstd (may be NULL) is kept for the gradients.  The gradients g_x and g_w may each be NULL; g_w
 * needs part_w, fp32 [amemRmsNormGradBlocks(rows)][dim] of work memory. */
ncclResult_t amemRmsNorm(const void* x, const void* w, void* y, float* rstd, long long rows, int dim, double eps, cudaStream_t stream);
int amemRmsNormGradBlocks(long long rows);
ncclResult_t amemRmsNormGrad(const void* g_y, const void* x, const void* w, const float* rstd, void* g_x, float* part_w, void* g_w, long long rows,
                             int dim, cudaStream_t stream);
/* Gradient of an embedding table, bf16 [rows, dim]: the sums of the rows of g[tokens, dim] that have the same id, fp32 inside, in an
 * order that the ids alone decide; zero where no token points.  The second form takes its work memory, `tokens` bytes rounded
 * up to 16 at a 16-byte boundary, from the caller; the first allocates it on the stream. */
ncclResult_t amemEmbeddingGrad(const void* g, const long long* ids, void* g_table, int tokens, int dim, long long rows, cudaStream_t stream);
ncclResult_t amemEmbeddingGradShared(const void* g, const long long* ids, void* g_table, void* work, int tokens, int dim, long long rows,
                                     cudaStream_t stream);
/* Rotary embedding of one or two bf16 tensors [batch, heads[i], seq, dim]: (o[2j], o[2j+1]) is (x[2j], x[2j+1]) turned by
 * the angle whose fp32 cosine and sine stand at [position][j] (by its negative with inverse != 0, which is the gradient).
 * strides: six per tensor, of batch, head and position in elements, first of the input, then of the output; multiples of
 * 8, the last dimension is dense. */
ncclResult_t amemRotate(const void* const* in, void* const* out, const int* heads, const long long* strides, int tensors, const float* cos,
                        const float* sin, int batch, int seq, int dim, int inverse, cudaStream_t stream);
/* dst[i][0 .. n[i]) += scale * src[i][0 .. n[i]) (fp32 += bf16) for every piece i; the pieces of dst do not overlap. */
ncclResult_t amemSumPieces(const void* const* src, float* const* dst, const long long* n, int pieces, double scale, cudaStream_t stream);
/* The same as an operation of a communicator of one rank: refused where that refuses one, and within its bound on blocks.  The plan says
 * how many blocks the largest of its launches runs where the user bounds them to block_cap (0: no bound); host arithmetic only. */
ncclResult_t amemSumPiecesLocal(const void* const* src, float* const* dst, const long long* n, int pieces, double scale, ncclComm_t comm,
                                cudaStream_t stream);
ncclResult_t amemSumPiecesPlan(const long long* n, int pieces, int block_cap, size_t* blocks);
/* Routing of T tokens, bf16 [T, d] (d a multiple of 8), over E <= 256 experts: the k largest products with the rows of
 * router, bf16 [E, d], rounded to bf16, largest first (equal ones by the lower expert), and the softmax over them: int32 and
 * fp32 [T, k].  The gradient of the weights down to the logits is bf16 [T, E]. */
ncclResult_t amemMoeRoute(const void* x, const void* router, int* topk_idx, float* topk_w, int T, int d, int E, int k, cudaStream_t stream);
ncclResult_t amemMoeRouteGrad(const float* g_w, const float* topk_w, const int* topk_idx, void* g_logits, int T, int E, int k, cudaStream_t stream);
/* On a communicator of one rank, the gradient of the tokens through dispatch and routing at once, bf16 [T, d]:
 * g_x[t] = sum_j g_rows[send_pos[t, j]] + g_logits[t, e_j] * router[e_j], e_j = topk_idx[t, j]. */
ncclResult_t amemMoeInputGradLocal(const void* g_rows, const int* send_pos, const int* topk_idx, const void* g_logits, const void* router, void* g_x,
                                   int rows, int T, int k, int d, int E, ncclComm_t comm, cudaStream_t stream);
/* One AdamW update of n parameters in one pass: fp32 gradient, moments and master weights, bf16 copy of the
 * new weights; step counts from 1. */
ncclResult_t amemAdamW(const float* grad, float* m, float* v, float* master, void* shard_bf16, long long n, double lr, double beta1, double beta2,
                       double eps, double weight_decay, long long step, cudaStream_t stream);
/* Refuses what an operation of the communicator would be refused for (paused, aborted, in error, another device
 * current) and orders the stream behind the communicator's previous one: for callers whose operation has
 * nothing to send, because the communicator has one rank, and who run it without the communicator. */
ncclResult_t amemCommBegin(ncclComm_t comm, cudaStream_t stream);
/* What amemGemmBf16 does for a problem on a GPU with `sms` SMs, operands and result 16-byte aligned: *form 2 =
 * few rows (*tile tokens, *slices 2 where tiles are cut along K), 1 = SM pairs (tiles of 256 x *tile, each cut
 * in *slices along K), 0 = the one-SM form (see amemGemmPlan).  Host arithmetic only; outputs may be NULL. */
ncclResult_t amemGemmForm(int M, int N, int K, int sms, int* form, int* tile, int* slices);
/* How the form for few rows shares out its blocks of K: *schedule 0 = whole tiles, 1 = all of them evenly over the SMs, 2 = a tile's owner
 * with its helpers; -1: amemGemmBf16 takes another form.  Host arithmetic only. */
ncclResult_t amemGemmSchedule(int M, int N, int K, int sms, int* schedule);
/* The tiling of the one-SM form of the GEMM (the fused all-gather GEMM's) for a GPU with `sms` SMs: tile
 * rows (128 or 256), tile columns, K-slices of the last wave (1 = not split).  Host arithmetic only;
 * outputs may be NULL. */
/* Variant (1 one-shot, 2 two-shot, 3 NVLS, 0 n/a), grid and chunk the library picks for a collective
 * (kind: 0 all-reduce, 1 all-gather, 2 reduce-scatter, 3 broadcast, 4 reduce, 5 all-to-all) on `nranks`
 * GPUs; stage_bytes 0 = default staging.  Host arithmetic only. */
ncclResult_t amemTunerPlan(int kind, size_t count, ncclDataType_t dtype, int nranks, int nvls, size_t stage_bytes, int* algo,
                           int* blocks, size_t* chunk_elems);
/* Blocks of the single-pass form of a collective on a communicator of one rank (*blocks; 0: the general kernel
 * runs) whose blocks the user bounds to block_cap (maxCTAs, AMEM_MAX_BLOCKS; 0: no bound).  Host arithmetic only. */
ncclResult_t amemLocalPlan(size_t count, ncclDataType_t dtype, ncclDataType_t out_dtype, float scale, int block_cap, size_t* blocks);
/* Debug guard behind the staging layout (AMEM_CANARY=1): ncclInternalError if a kernel wrote past it. */
/* Variable-size all-to-all; counts and displacements in elements, MPI_Alltoallv convention. */
ncclResult_t amemAlltoAllv(const void* sendbuff, const size_t* sendcounts, const size_t* sdispls, void* recvbuff,
                           const size_t* recvcounts, const size_t* rdispls, ncclDataType_t datatype, ncclComm_t comm, cudaStream_t stream);
ncclResult_t amemCheckCanary(ncclComm_t comm);
ncclResult_t amemDebugDirtyCanary(ncclComm_t comm); /* test hook: dirties the guard */
/* Grouped GEMM (one launch for all experts of a rank): for every group e,
 * C[group_off[e] .. group_off[e+1], :] = A[same rows, :] * B[e]^T.  group_off is a DEVICE array of
 * groups + 1 int32 row offsets (amemMoeDispatch's expert_offsets), B is bf16 [groups, N, K].
 * epilogue 0: C is bf16 [rows_cap, N]; epilogue 1 (SwiGLU): B[e]'s rows alternate in blocks of 32
 * gate rows and 32 up rows and C is bf16 [rows_cap, N / 2] = silu(gate) * up. */
ncclResult_t amemGroupedGemmBf16(const void* A, const void* B, void* C, const int* group_off, int groups, int rows_cap, int rows_hint,
                                 int N, int K, int epilogue, cudaStream_t stream);
/* The gradients of the grouped product, from the operands as they lie: amemGroupedGemmBf16Input gives
 * C[rows of e, K] = A[rows of e, N] * B[e] (B bf16 [groups, N, K]); amemGroupedGemmBf16Weight gives
 * C[e] = A[rows of e]^T * B[rows of e], bf16 [groups, N, K], zeros for a group without rows. */
ncclResult_t amemGroupedGemmBf16Input(const void* A, const void* B, void* C, const int* group_off, int groups, int rows_cap, int rows_hint,
                                      int N, int K, cudaStream_t stream);
ncclResult_t amemGroupedGemmBf16Weight(const void* A, const void* B, void* C, const int* group_off, int groups, int rows_cap, int N, int K,
                                       cudaStream_t stream);
ncclResult_t amemGemmPlan(int M, int N, int K, int sms, int* tile_rows, int* tile_cols, int* tail_slices);
/* Schedule of amemAllGatherGemm for nranks ranks (1 = mover warps in every CTA, 0 = dedicated mover CTAs), rows of a
   shard per ready flag and ready flags per source rank.  Host arithmetic, no GPU needed. */
ncclResult_t amemAllGatherGemmPlan(int nranks, int rows_per_rank, int K, int* mover_warps, int* rows_per_flag, int* flags_per_rank);
/* One kernel: C[M,N] = allgather_rows(a_shard)[M,K] * B[N,K]^T.  a_shard holds this rank's
 * M/nranks rows; the transfer of the other ranks' rows overlaps the tensor-core work. */
ncclResult_t amemAllGatherGemm(const void* a_shard, const void* B, void* C, int M, int N, int K, ncclComm_t comm, cudaStream_t stream);
/* One kernel: out[M/nranks,N] = reduce_scatter_rows(A[M,K] * B[N,K]^T); partial tiles travel
 * to their owner from the epilogue and are summed there in rank order. */
ncclResult_t amemGemmReduceScatter(const void* A, const void* B, void* out, int M, int N, int K, ncclComm_t comm, cudaStream_t stream);
/* MoE expert parallelism.  Experts are spread evenly over the communicator (expert e lives on
 * rank e / (E / nranks)).  amemMoeBuffers (collective) returns this rank's receive buffer and
 * expert-output buffer, both bf16 [capacity_rows, d] in symmetric scratch memory.
 * amemMoeDispatch writes every (token, choice) row into its expert's rank at its final
 * expert-sorted position (the permutation is fused into the all-to-all); amemMoeCombine pulls
 * the expert outputs back and applies the routing weights in one pass. */
ncclResult_t amemMoeBuffers(ncclComm_t comm, int capacity_rows, int d, void** recv_x, void** y);
/* Whether a communicator of one rank gathers the combine's rows by bulk copies (*streams 1) or by the warps' own loads (0).  Host
 * arithmetic only. */
ncclResult_t amemMoeCombinePlan(int T, int k, int d, int* streams);
/* The same on a communicator of one rank between the caller's own buffers, and the combine's backward:
 * g_y[row(t, j)] = topk_w[t, j] * g_out[t] (bf16), g_w[t, j] = <g_out[t], y[row(t, j)]> (fp32). */
ncclResult_t amemMoeDispatchLocal(const void* x, const int* topk_idx, int T, int k, int d, int E, void* recv, int capacity_rows, int* expert_counts,
                                  int* expert_offsets, int* send_pos, int* dropped_rows, ncclComm_t comm, cudaStream_t stream);
ncclResult_t amemMoeCombineLocal(const int* topk_idx, const float* topk_w, const int* send_pos, const void* y, int rows, void* out, int T, int k, int d, int E,
                                 ncclComm_t comm, cudaStream_t stream);
ncclResult_t amemMoeCombineGradLocal(const void* g_out, const void* y, const float* topk_w, const int* send_pos, void* g_y, float* g_w, int rows, int T, int k,
                                     int d, ncclComm_t comm, cudaStream_t stream);
ncclResult_t amemMoeDispatch(const void* x, const int* topk_idx, int T, int k, int d, int E, int capacity_rows, int* expert_counts,
                             int* expert_offsets, int* send_pos, ncclComm_t comm, cudaStream_t stream);
/* The same with one more output: *dropped_rows (device int, may be null) = rows routed to this rank
 * that did not fit capacity_rows.  Such rows are not sent (send_pos -1, weight zero in the combine),
 * the counts and offsets describe only stored rows, and the communicator stays usable. */
ncclResult_t amemMoeDispatchCounted(const void* x, const int* topk_idx, int T, int k, int d, int E, int capacity_rows, int* expert_counts,
                                    int* expert_offsets, int* send_pos, int* dropped_rows, ncclComm_t comm, cudaStream_t stream);
ncclResult_t amemMoeCombine(const int* topk_idx, const float* topk_w, const int* send_pos, void* out, int T, int k, int d, int E,
                            int capacity_rows, ncclComm_t comm, cudaStream_t stream);
/* 1 if the communicator's ranks share one GPU and run as one cooperative grid; 1 if NVLS is in use. */
ncclResult_t amemCommInfo(ncclComm_t comm, int* emulated, int* nvls, size_t* stage_bytes);
/* Host-side fault injection for tests: what = "uds:drop" | "uds:short" | "uds:nofd" |
 * "uds:delay" | "uds:clear" | "vmm:create" | "vmm:map" | "vmm:import" | "vmm:export" |
 * "vmm:host_alloc"; the nth next such call misbehaves. */
ncclResult_t amemInject(const char* what, int nth, int param);
/* Bytes of physical memory and number of mappings this process holds through the backend. */
ncclResult_t amemBackendUsage(size_t* physical_bytes, size_t* mappings, const char** backend_name);
/* Runs one device thread that waits, as the collective kernels wait for their peers, for a word that
 * is set beforehand (flag_is_set != 0) or never (0), for at most timeout_ms.  *code receives the
 * device error code written to host-visible status words (0 = the flag came, 1 = the wait ran out),
 * *waited_ms the kernel's duration.  The kernel always returns; the CUDA context stays usable. */
ncclResult_t amemDeviceWaitProbe(int timeout_ms, int flag_is_set, int* code, float* waited_ms);
/* 1 when the memory backend is CUDA device memory, 0 for the host-memory mock. */
int amemBackendIsDevice(void);
/* JSON with the time spent in every kind of VMM driver call (create, map, set_access, ...). */
ncclResult_t amemBackendTimings(char* buf, size_t len, int reset);
const char* amemLastError(void);

#ifdef __cplusplus
}
#endif
#endif /* AMEM_B200_NCCL_H_ */
