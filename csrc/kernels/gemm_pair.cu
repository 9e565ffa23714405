// tcgen05 GEMM on pairs of SMs (cta_group::2).
//
// A cluster of two CTAs computes tiles of 256 x bn (bn <= 256): each CTA loads its own 128 rows of
// A and HALF of the columns of B, the tensor cores of both SMs read both halves, and each CTA keeps
// the accumulator of its 128 rows in its own tensor memory.  Against 128 x 256 tiles on one SM that
// is a third less shared memory filled per product (32 KB instead of 48 KB per 64 of K), which is
// what bounds the one-SM form; six stages fit, and with 256 of 512 TMEM columns per tile the
// epilogue of one tile runs under the main loop of the next.  TMA loads carry no multicast.
//
// Roles per CTA: warp 0 loads, warp 1 of the even CTA issues every MMA, warps 2-5 drain TMEM, and for groups
// along K warp 6 clears the rows of a group's last block that belong to the next group.  The
// `full` barrier of a stage lives in the even CTA and counts the bytes of both; `empty` and the
// accumulator's `tfull` are signalled in both CTAs by one commit.
//
// A product with fewer tiles than half of the SM pairs is cut along K: the slices of a tile exchange
// fp32 partial sums through a workspace, each slice sums its share of the tile's 32-column chunks over
// all slices, in slice order (so the result does not depend on who comes first).
//
// Result rows leave through a small swizzled staging area per warp, so that a warp's store covers
// whole 128-byte lines (one thread per row would touch 32 lines with 16 bytes each).
//
// Measured (B200, back to back in a graph, us; one-SM kernel -> this one): 2048 x 8192 x 2048 62.6 -> 47.5,
// 1000 x 3584 x 8192 58.2 -> 44.5, 512 x 28672 x 4096 106.7 -> 92.9, 500 x 4096 x 14336 67 -> 52,
// 4096^3 101.5 -> 95.0; 4096 x 28672 x 4096 alone 648 -> 588 (1.64 PFLOP/s).  Long runs of the largest
// products end at the power limit, where both forms and cuBLAS meet (8192 x 7168 x 8192: 752 - 769).
//
// Every wait is bounded and ends in an error status.
#include <algorithm>

#include "../core/log.h"
#include "coll_device.cuh"
#include "gemm_pair.h"
#include "pdl.cuh"
#include "sm100_prims.cuh"
#include "smem_limit.h"

namespace amem {
namespace pairk {

using namespace sm100;

constexpr int HM = 128;            // rows of A per CTA
constexpr int TM = 2 * HM;         // rows of a tile
constexpr int BN_MAX = 256, BK = 64;
constexpr int STAGES = 6;
constexpr int A_BYTES = HM * BK * 2, B_BYTES = (BN_MAX / 2) * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int CHUNK_BYTES = 64 * BK * 2;     // MN-major operands: 64 columns x 64 of K per TMA box
constexpr int EPI_WARPS = 4, EPI_BYTES = 32 * 128;   // staging of one epilogue warp: 32 rows x 128 bytes
constexpr int THREADS = 32 * (2 + EPI_WARPS), CLEAR_WARP = 2 + EPI_WARPS;
constexpr int MAX_GROUPS = 256;
constexpr int MAX_SLICES = 8;                        // 32-column chunks of the widest tile: one per slice at least
constexpr size_t SLOT_FLOATS = (size_t)HM * BN_MAX;  // partial sums of one CTA
constexpr uint32_t PIECE_BYTES = HM * 32 * 4;        // one 32-column chunk of them
constexpr uint32_t TMEM_COLS = 512;

struct Params {
  void* C;
  int M, N, K, bn, ldc;
  int mode, epilogue, groups;
  const int* group_off;
  uint32_t* status;
  unsigned long long timeout_ns;
  int slices;        // plain: cuts of every tile along K (one item of work per pair then), 1: none
  float* sk_ws;      // [tile][slice][CTA of the pair][4-column group][128 rows][4]
  uint32_t* sk_ctr;  // [tile][CTA of the pair]{arrived, finished}
};

struct __align__(8) Ctl {
  uint64_t full[STAGES];    // used in the even CTA
  uint64_t empty[STAGES];
  uint64_t tfull[2];
  uint64_t tempty[2];       // used in the even CTA
  uint64_t tail;            // the exchanged partial sums have landed in this CTA
  uint64_t ragged[STAGES];  // the ragged last K block of a group has landed in this CTA
  uint32_t tmem_base;
  int abort;
  int off[MAX_GROUPS + 1];        // group offsets, made monotonic
  int first_tile[MAX_GROUPS + 1]; // tiles before group e
};

// ---- cluster primitives
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the even CTA's copy of a control word
__device__ __forceinline__ uint32_t in_leader(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
__device__ __forceinline__ void arrive_leader(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// counts bytes as landed on the even CTA's barrier: what this CTA wrote before is visible to whoever waits there
__device__ __forceinline__ void complete_leader(uint32_t bar, uint32_t bytes) {
  asm volatile("fence.acq_rel.cluster;" ::: "memory");
  asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const void* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void commit_pair(uint64_t* bar) {   // arrives at the same barrier of both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Bounded wait of a whole warp (false: gave up).
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, unsigned long long timeout_ns, volatile int* abort) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, timeout_ns, abort));
}
// Operand tile stored with its M or N index contiguous: chunks of 64 of that index, each 64 rows (of
// K) of 128 bytes in the 128-byte swizzle; chunks are CHUNK_BYTES apart, groups of 8 rows 1024 bytes.
__device__ __forceinline__ uint64_t make_smem_desc_mn_sw128(const void* tile) {
  uint64_t addr = (uint64_t)(smem_u32(tile) & 0x3FFFF) >> 4;
  return addr | ((uint64_t)(CHUNK_BYTES >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// Only operands that both lie by their contraction index can have groups along it, and need the warp that clears.
constexpr int threads_of(int a_mn, int b_mn) { return THREADS + (a_mn && b_mn ? 32 : 0); }

struct Tile {
  int group, m0, n_blk;   // first row of the tile inside the group (or matrix), column block
  int rows;               // rows left from m0 on (may exceed a tile)
  int row_base;           // grouped rows: the group's first row in A and C
  int k0, nk;             // first contraction index and their number
  int slice;
};

__device__ __forceinline__ int tiles_of(const Params& p, const Ctl* c, int e, int tiles_n) {
  if (p.mode == kPairGroupedRows) return ((c->off[e + 1] - c->off[e] + TM - 1) / TM) * tiles_n;
  return ((p.M + TM - 1) / TM) * tiles_n;
}

template <int CUT>
__device__ __forceinline__ Tile tile_at(const Params& p, const Ctl* c, int item, int tiles_n) {
  const int t = CUT ? item / p.slices : item;
  int e = 0, hi = p.groups;
  while (hi - e > 1) {   // last group that starts at or before t
    const int mid = (e + hi) / 2;
    if (c->first_tile[mid] <= t) e = mid;
    else hi = mid;
  }
  const int v = t - c->first_tile[e];
  const bool ragged_m = p.mode == kPairGroupedRows;
  const int rows = ragged_m ? c->off[e + 1] - c->off[e] : p.M;
  const int tiles_m = (rows + TM - 1) / TM;
  // Bands of 8 row tiles, rows fastest inside: the ~74 tiles in flight then cover about 8 x 9 tiles
  // and re-use both operands out of L2.
  const int GM = 8;
  const int band = v / (GM * tiles_n), first = band * GM;
  const int gm = min(GM, tiles_m - first);
  const int w = v - band * GM * tiles_n;
  Tile o;
  o.group = e;
  const int m_blk = first + w % gm;
  o.n_blk = w / gm;
  o.m0 = m_blk * TM;
  o.rows = rows - o.m0;
  o.row_base = ragged_m ? c->off[e] : 0;
  o.k0 = p.mode == kPairGroupedK ? c->off[e] : 0;
  o.nk = p.mode == kPairGroupedK ? c->off[e + 1] - c->off[e] : p.K;
  o.slice = 0;
  if (CUT) {
    o.slice = item - t * p.slices;
    const int kbs = (p.K + BK - 1) / BK;
    const int lo = o.slice * kbs / p.slices, hi2 = (o.slice + 1) * kbs / p.slices;
    o.k0 = lo * BK;
    o.nk = min(p.K, hi2 * BK) - o.k0;
  }
  return o;
}

// CUT: tiles may be cut along K (kept apart: the sum over slices costs registers)
template <int A_MN, int B_MN, int CUT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(threads_of(A_MN, B_MN), 1)
pair_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b) {
  extern __shared__ char smem_raw[];
  char* ring = (char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  char* staging = ring + STAGES * STAGE_BYTES;
  Ctl* ctl = (Ctl*)(staging + EPI_WARPS * EPI_BYTES);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x / 32, 0), lane = threadIdx.x % 32;   // warp: known to be uniform
  const uint32_t rank = cluster_rank();
  const int cluster = blockIdx.x / 2, clusters = gridDim.x / 2;
  volatile int* abort = &ctl->abort;
  const int bn = p.bn, half = bn / 2;
  pdl_launch_dependents();

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&ctl->full[s], 1);    // the even CTA arrives, with the byte count of both
      mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ctl->tfull[b], 1);
      mbar_init(&ctl->tempty[b], 2 * EPI_WARPS);
    }
    mbar_init(&ctl->tail, 1);
    for (int s = 0; s < STAGES; ++s) mbar_init(&ctl->ragged[s], 1);
    ctl->abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl->tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_wait();   // from here on: what earlier kernels wrote is read, what they read may be overwritten
  const int out_cols = p.epilogue == kPairStore ? p.N : p.N / 2;
  const int tiles_n = (p.N + bn - 1) / bn;
  if (warp == 2) {
    // group table in shared memory: offsets and tiles before each group
    if (p.mode == kPairPlain) {
      if (lane == 0) {
        ctl->off[0] = 0;
        ctl->off[1] = p.M;
        ctl->first_tile[0] = 0;
        ctl->first_tile[1] = tiles_of(p, ctl, 0, tiles_n);
      }
    } else {
      const int limit = p.mode == kPairGroupedRows ? p.M : p.K;
      int carry = 0, last = 0;
      for (int e0 = 0; e0 <= p.groups; e0 += 32) {
        const int e = e0 + lane;
        int v = e <= p.groups ? min(max(p.group_off[e], 0), limit) : 0;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {   // running maximum: offsets never step back
          const int o = __shfl_up_sync(0xffffffffu, v, d);
          if (lane >= d) v = max(v, o);
        }
        v = max(v, last);
        last = __shfl_sync(0xffffffffu, v, 31);
        if (e <= p.groups) ctl->off[e] = v;
      }
      __syncwarp();
      for (int e0 = 0; e0 < p.groups; e0 += 32) {
        const int e = e0 + lane;
        int n = e < p.groups ? tiles_of(p, ctl, e, tiles_n) : 0;
        int s = n;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
          const int o = __shfl_up_sync(0xffffffffu, s, d);
          if (lane >= d) s += o;
        }
        if (e < p.groups) ctl->first_tile[e] = carry + s - n;
        carry += __shfl_sync(0xffffffffu, s, 31);
      }
      if (lane == 0) ctl->first_tile[p.groups] = carry;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();   // the partner's barriers are initialised before anything is signalled there
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;
  const int total = ctl->first_tile[p.groups] * (CUT ? p.slices : 1);

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const int b_chunks = (half + 63) / 64;
    const uint32_t bytes = (uint32_t)(A_BYTES + (B_MN ? b_chunks * CHUNK_BYTES : half * BK * 2));
    for (int t = cluster; t < total && ok; t += clusters) {
      const Tile tl = tile_at<CUT>(p, ctl, t, tiles_n);
      const int a_row = tl.row_base + tl.m0 + (int)rank * HM;
      int b_row = tl.n_blk * bn + (int)rank * half;
      if (p.epilogue == kPairSwiGLUHalves) b_row = tl.n_blk * half + (int)rank * (p.N / 2);
      const int b_z = p.mode == kPairGroupedRows ? tl.group : 0;
      const int num_kb = (tl.nk + BK - 1) / BK;
      for (int kb = 0; kb < num_kb && ok; ++kb) {
        char* sa = ring + (size_t)stage * STAGE_BYTES;
        char* sb = sa + A_BYTES;
        const int k = tl.k0 + kb * BK;
        // The last K block of a group may reach into the next group's rows (both operands hold rows
        // there): it lands on a barrier of this CTA first, where another warp clears those rows and counts it.
        // (Done here, the loads behind it waited: 149 us for 8 x 1024 rows of 3072 x 4096, 190 for groups of about
        // that size, 177 so: their row tiles and K blocks are not whole.)
        const bool clear = A_MN && B_MN && p.mode == kPairGroupedK && tl.nk - kb * BK < BK;
        ok = ok && wait_bar(&ctl->empty[stage], phase ^ 1u, p.timeout_ns, abort);
        if (ok) {
          if (elect_one()) {
            // Only the even CTA arrives (an arrival from the odd one would have to be a release at
            // cluster scope, which costs half a microsecond per stage); bytes may land before it does.
            if (rank == 0) mbar_expect_tx(&ctl->full[stage], 2 * bytes);
            uint32_t bar = in_leader(&ctl->full[stage]);
            if (clear) {
              bar = smem_u32(&ctl->ragged[stage]);
              mbar_expect_tx(&ctl->ragged[stage], bytes);
            }
            if (A_MN) {
#pragma unroll
              for (int c = 0; c < HM / 64; ++c) tma_load_3d_pair(sa + c * CHUNK_BYTES, &map_a, bar, a_row + c * 64, k, 0);
            } else {
              tma_load_3d_pair(sa, &map_a, bar, k, a_row, 0);
            }
            if (B_MN) {
              for (int c = 0; c < b_chunks; ++c) tma_load_3d_pair(sb + c * CHUNK_BYTES, &map_b, bar, b_row + c * 64, k, b_z);
            } else {
              tma_load_3d_pair(sb, &map_b, bar, k, b_row, b_z);
            }
          }
          __syncwarp();
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    // every stage handed back: no signal of the partner's is still on its way to this CTA's barriers
    for (int s = 0; s < STAGES && ok; ++s) {
      ok = wait_bar(&ctl->empty[stage], phase ^ 1u, p.timeout_ns, abort);
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (!ok) {
      // gave up: copies that are still in flight land within microseconds; wait for them before leaving
      const unsigned long long t0 = gtimer_ns();
      while (gtimer_ns() - t0 < 2000000ull) {
      }
    }
  } else if (A_MN && B_MN && warp == CLEAR_WARP) {
    // ------------------------------------------------------------ rows of the next group out of a group's last block
    if (p.mode == kPairGroupedK) {
      int stage = 0;
      uint32_t phases = 0;      // of ragged[], a bit each
      bool ok = true;
      const int b_chunks = (half + 63) / 64;
      const uint32_t bytes = (uint32_t)(A_BYTES + b_chunks * CHUNK_BYTES);
      for (int t = cluster; t < total && ok; t += clusters) {
        const Tile tl = tile_at<CUT>(p, ctl, t, tiles_n);
        const int num_kb = (tl.nk + BK - 1) / BK;
        if (num_kb == 0) continue;
        const int at = (stage + num_kb - 1) % STAGES, r0 = tl.nk - (num_kb - 1) * BK;
        stage = (stage + num_kb) % STAGES;
        if (r0 == BK) continue;
        ok = wait_bar(&ctl->ragged[at], phases >> at & 1u, p.timeout_ns, abort);
        phases ^= 1u << at;
        if (!ok) break;
        char* sa = ring + (size_t)at * STAGE_BYTES;
        const int r1 = (r0 + 15) & ~15;   // the MMAs of this block read r1 rows
        const int lines = (r1 - r0) * (HM / 64 + b_chunks);
        for (int i = lane; i < lines * 8; i += 32) {
          const int l = i / 8, c = l / (r1 - r0), r = r0 + l % (r1 - r0);
          *(uint4*)(sa + c * CHUNK_BYTES + r * 128 + (i % 8) * 16) = make_uint4(0, 0, 0, 0);   // B's chunks follow A's
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) complete_leader(in_leader(&ctl->full[at]), bytes);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (even CTA)
    if (rank == 0) {
      const uint32_t idesc = make_idesc_bf16(TM, bn) | ((uint32_t)A_MN << 15) | ((uint32_t)B_MN << 16);
      const uint64_t da = A_MN ? make_smem_desc_mn_sw128(ring) : make_smem_desc_sw128(ring);
      const uint64_t db = B_MN ? make_smem_desc_mn_sw128(ring + A_BYTES) : make_smem_desc_sw128(ring + A_BYTES);
      int stage = 0, it = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = cluster; t < total && ok; t += clusters) {
        const Tile tl = tile_at<CUT>(p, ctl, t, tiles_n);
        if (tl.nk == 0) continue;   // an empty group: the epilogue writes zeros by itself
        const int buf = it & 1;
        ok = wait_bar(&ctl->tempty[buf], (((uint32_t)it >> 1) & 1u) ^ 1u, p.timeout_ns, abort);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t d = tmem_base + (uint32_t)(buf * BN_MAX);
        const int num_kb = (tl.nk + BK - 1) / BK;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = wait_bar(&ctl->full[stage], phase, p.timeout_ns, abort);
          if (!ok) break;
          tc_fence_after_sync();
          // The whole warp walks the loop and one elected thread issues: the descriptors then live in
          // uniform registers (issued from inside a one-thread branch the same loop took 1.5x as long).
          if (elect_one()) {
            const uint64_t at = (uint64_t)(stage * (STAGE_BYTES >> 4));
            // 16 of K: 32 bytes along a K-major row, or 16 rows of 128 bytes
            const int left = tl.nk - kb * BK;
            if (left >= BK) {
#pragma unroll
              for (int kk = 0; kk < BK / 16; ++kk)
                mma_pair(d, da + at + (uint64_t)(kk * (A_MN ? 128 : 2)), db + at + (uint64_t)(kk * (B_MN ? 128 : 2)), idesc, (kb | kk) ? 1u : 0u);
            } else {
#pragma unroll 1
              for (int kk = 0; kk < (left + 15) / 16; ++kk)
                mma_pair(d, da + at + (uint64_t)(kk * (A_MN ? 128 : 2)), db + at + (uint64_t)(kk * (B_MN ? 128 : 2)), idesc, (kb | kk) ? 1u : 0u);
            }
            commit_pair(&ctl->empty[stage]);
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (ok && elect_one()) commit_pair(&ctl->tfull[buf]);
        __syncwarp();
        ++it;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ epilogue
    const int lane_grp = warp % 4;                  // TMEM lanes [32 * lane_grp, +32)
    char* stg = staging + (warp - 2) * EPI_BYTES;
    const int sw = lane & 7;
    int it = 0;
    bool ok = true;
    for (int t = cluster; t < total && ok; t += clusters) {
      const Tile tl = tile_at<CUT>(p, ctl, t, tiles_n);
      const int r_first = (int)rank * HM + lane_grp * 32;    // first row of this warp inside the tile
      const int rows = min(32, tl.rows - r_first);           // rows to store (<= 0: none)
      const size_t c_row = (size_t)(p.mode == kPairGroupedK ? (size_t)tl.group * p.M : (size_t)tl.row_base) + tl.m0 + r_first;
      const bool swiglu = p.epilogue != kPairStore;
      const int col0 = tl.n_blk * (swiglu ? half : bn);
      const int cols = min(swiglu ? half : bn, out_cols - col0);
      __nv_bfloat16* C = (__nv_bfloat16*)p.C + c_row * (size_t)p.ldc + col0;
      if (tl.nk == 0) {
        for (int i = lane; i < max(rows, 0) * (cols / 8); i += 32)
          *(uint4*)(C + (size_t)(i / (cols / 8)) * p.ldc + (i % (cols / 8)) * 8) = make_uint4(0, 0, 0, 0);
        continue;
      }
      const int buf = it & 1;
      ok = wait_bar(&ctl->tfull[buf], ((uint32_t)it >> 1) & 1u, p.timeout_ns, abort);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t acc = tmem_base + (uint32_t)(buf * BN_MAX) + ((uint32_t)(lane_grp * 32) << 16);
      const int S = CUT ? p.slices : 1;
      const int second = p.epilogue == kPairSwiGLUHalves ? half : 0;   // columns of the up projection (split form)
      if (S > 1) {
        // hand the other slices their chunks: chunk number j of the result belongs to slice j % S
        float4* mine = (float4*)(p.sk_ws + ((size_t)(t / S * S + tl.slice) * 2 + rank) * SLOT_FLOATS) + lane_grp * 32 + lane;
        for (int cc = 0; cc < cols; cc += 32) {
          if ((cc / 32) % S == tl.slice) continue;
          for (int part = 0; part <= (second ? 1 : 0); ++part) {
            uint32_t v[32];
            tmem_ld_32x32(acc + (uint32_t)(cc + part * second), v);
            tmem_ld_wait();
            float4* dst = mine + (size_t)((cc + part * second) / 4) * HM;
#pragma unroll
            for (int q = 0; q < 8; ++q)
              dst[(size_t)q * HM] = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
          }
        }
        __threadfence();
        asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");
        uint32_t* ctr = p.sk_ctr + (size_t)(t / S * 2 + (int)rank) * 2;
        bool met = true;
        if (warp == 2 && lane == 0) {
          atomicAdd(ctr, 1u);
          met = dev::wait_flag_ge(ctr, (uint32_t)S, p.timeout_ns);
          __threadfence();
          if (met) {
            // the other slices' parts of this slice's chunks, all in flight at once, into the idle operand
            // ring (this pair has no other tile): 16 KB a piece, at most most_pieces() of them
            asm volatile("fence.proxy.async;" ::: "memory");
            const int n = ((cols + 31) / 32 - tl.slice + S - 1) / S * (second ? 2 : 1) * (S - 1);
            mbar_expect_tx(&ctl->tail, (uint32_t)n * PIECE_BYTES);
            char* dst = ring;
            for (int cc = tl.slice * 32; cc < cols; cc += S * 32)
              for (int part = 0; part <= (second ? 1 : 0); ++part)
                for (int s = 0; s < S; ++s) {
                  if (s == tl.slice) continue;
                  const float* src = p.sk_ws + ((size_t)(t / S * S + s) * 2 + rank) * SLOT_FLOATS + (size_t)((cc + part * second) / 4) * HM * 4;
                  bulk_load(dst, src, PIECE_BYTES, &ctl->tail);
                  dst += PIECE_BYTES;
                }
          }
        }
        met = __shfl_sync(0xffffffffu, met ? 1 : 0, 0) != 0;
        ok = met && wait_bar(&ctl->tail, 0, p.timeout_ns, abort);
        if (!met) *abort = 1;   // (the other warps' wait then ends as well)
        if (!ok) break;
      }
      const char* piece_at = ring;
      // the sum of columns [cc, cc + 32) of this lane's row over all slices, in slice order
      auto read_chunk = [&](int cc, uint32_t (&v)[32]) {
        tmem_ld_32x32(acc + (uint32_t)cc, v);
        tmem_ld_wait();
        if (S > 1) {
          float sum[32];
#pragma unroll
          for (int q = 0; q < 32; ++q) sum[q] = 0.f;
#pragma unroll 1
          for (int s = 0; s < S; ++s) {
            if (s == tl.slice) {
#pragma unroll
              for (int q = 0; q < 32; ++q) sum[q] += __uint_as_float(v[q]);
              continue;
            }
            const float4* x = (const float4*)piece_at + lane_grp * 32 + lane;
            piece_at += PIECE_BYTES;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const float4 f = x[q * HM];
              sum[4 * q] += f.x;
              sum[4 * q + 1] += f.y;
              sum[4 * q + 2] += f.z;
              sum[4 * q + 3] += f.w;
            }
          }
#pragma unroll
          for (int q = 0; q < 32; ++q) v[q] = __float_as_uint(sum[q]);
        }
      };
      // one pass = 64 result columns: every lane converts its row, then the warp stores 4 rows x 128 bytes at a time
      for (int c = 0; c < cols; c += 64) {
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          const int cc = c + h * 32;
          if (cc < cols && (S == 1 || (cc / 32) % S == tl.slice)) {
            alignas(16) __nv_bfloat162 r[16];
            if (!swiglu) {
              uint32_t v[32];
              read_chunk(cc, v);
#pragma unroll
              for (int q = 0; q < 16; ++q) r[q] = __floats2bfloat162_rn(__uint_as_float(v[2 * q]), __uint_as_float(v[2 * q + 1]));
            } else {
              uint32_t g[32], u[32];
              read_chunk(second ? cc : 2 * cc, g);
              read_chunk(second ? cc + second : 2 * cc + 32, u);
              if (lane >= rows) {   // zeros of rows that are none would send the quotient down its slow path, and the warp with it
#pragma unroll
                for (int q = 0; q < 32; ++q) g[q] = __float_as_uint(1.f);
              }
#pragma unroll
              for (int q = 0; q < 16; ++q) {
                const float g0 = __uint_as_float(g[2 * q]), g1 = __uint_as_float(g[2 * q + 1]);
                r[q] = __floats2bfloat162_rn(g0 / (1.f + __expf(-g0)) * __uint_as_float(u[2 * q]),
                                             g1 / (1.f + __expf(-g1)) * __uint_as_float(u[2 * q + 1]));
              }
            }
            // 16-byte pieces are placed by (piece ^ row): neither the row-wise writes nor the line-wise reads conflict
#pragma unroll
            for (int j = 0; j < 4; ++j) *(uint4*)(stg + lane * 128 + (((h * 4 + j) ^ sw) * 16)) = ((const uint4*)r)[j];
          }
        }
        __syncwarp();
        const int piece = lane & 7, my_chunk = (c + piece * 8) / 32;
        if (c + piece * 8 < cols && (S == 1 || my_chunk % S == tl.slice)) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int row = i * 4 + lane / 8;
            if (row < rows) *(uint4*)(C + (size_t)row * p.ldc + c + piece * 8) = *(const uint4*)(stg + row * 128 + ((piece ^ (row & 7)) * 16));
          }
        }
        __syncwarp();
      }
      if (S > 1) {
        asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");   // this CTA has read all it needs
        uint32_t* ctr = p.sk_ctr + (size_t)(t / S * 2 + (int)rank) * 2;
        if (warp == 2 && lane == 0) {
          __threadfence();
          if (atomicAdd(ctr + 1, 1u) == (uint32_t)S - 1u) {   // the last reader leaves the counters at zero
            ctr[0] = 0;
            ctr[1] = 0;
            __threadfence();
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive_leader(in_leader(&ctl->tempty[buf]));
      ++it;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x == 0 && *abort) dev::report_error(p.status, kDevGemmTimeout, 0, 0, (int)blockIdx.x, 0xdead0010u);
  cluster_sync();   // neither CTA leaves while the other may still read or signal its shared memory
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

constexpr size_t kSmemBytes = (size_t)STAGES * STAGE_BYTES + EPI_WARPS * EPI_BYTES + sizeof(Ctl) + 1024;
static_assert(A_BYTES == (HM / 64) * CHUNK_BYTES, "B's chunks follow A's without a gap");
// Pieces of 32 columns that a slice collects: its share of the chunks, rounded up, from every other slice (12 for
// 7 slices of a 256-wide tile, of which the first has chunks 0 and 7).  A SwiGLU tile has half the chunks, in two parts,
// and at most a slice for each of them.
constexpr int most_pieces() {
  int most = 0;
  for (int s = 2; s <= MAX_SLICES; ++s) {
    const int chunks = BN_MAX / 32, n = (chunks + s - 1) / s * (s - 1), n_swiglu = s <= chunks / 2 ? 2 * ((chunks / 2 + s - 1) / s) * (s - 1) : 0;
    most = n > most ? n : most;
    most = n_swiglu > most ? n_swiglu : most;
  }
  return most;
}
static_assert((size_t)most_pieces() * PIECE_BYTES <= (size_t)STAGES * STAGE_BYTES, "the exchanged chunks must fit the operand ring");
static_assert(kSmemBytes <= 227 * 1024, "operand ring, staging and control words must fit one SM's shared memory");

template <int A_MN, int B_MN, int CUT>
Status launch_one(const Params& p, const CUtensorMap& ma, const CUtensorMap& mb, int grid, cudaStream_t stream) {
  static OncePerDevice raised;
  cudaError_t e = allow_smem(raised, pair_kernel<A_MN, B_MN, CUT>, kSmemBytes);
  if (e != cudaSuccess) return fail(kCudaError, "cudaFuncSetAttribute(%zu bytes of shared memory): %s", kSmemBytes, cudaGetErrorString(e));
  e = launch_overlapped(pair_kernel<A_MN, B_MN, CUT>, dim3(grid), dim3(threads_of(A_MN, B_MN)), kSmemBytes, stream, p, ma, mb);
  if (e != cudaSuccess) return fail(kCudaError, "pair gemm launch failed: %s", cudaGetErrorString(e));
  return kSuccess;
}

template <int A_MN, int B_MN>
Status launch(const Params& p, const CUtensorMap& ma, const CUtensorMap& mb, int grid, cudaStream_t stream) {
  return p.slices > 1 ? launch_one<A_MN, B_MN, 1>(p, ma, mb, grid, stream) : launch_one<A_MN, B_MN, 0>(p, ma, mb, grid, stream);
}

}  // namespace pairk

// [z][outer][inner] bf16 array with a box of box_inner x box_outer
Status make_bf16_map(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t z, uint32_t box_outer) {
  typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static EncodeFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return (EncodeFn)f;
  }();
  if (!fn) return fail(kCudaError, "cuTensorMapEncodeTiled is not available in this driver");
  if (((uintptr_t)base & 15) || inner % 8) return fail(kInvalidArgument, "TMA needs a 16-byte aligned base and row pitch");
  cuuint64_t dims[3] = {inner, outer, z};
  cuuint64_t strides[2] = {inner * 2, inner * outer * 2};
  cuuint32_t box[3] = {64, box_outer, 1}, estr[3] = {1, 1, 1};
  auto encode = [&] {
    return fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {   // a thread that has made no CUDA call yet (an autograd engine's)
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = encode();
  }
  if (r != CUDA_SUCCESS) return fail(kCudaError, "cuTensorMapEncodeTiled failed: %d (inner %llu outer %llu z %llu)", (int)r, (unsigned long long)inner,
                                     (unsigned long long)outer, (unsigned long long)z);
  return kSuccess;
}

int pair_gemm_pick_bn(long row_tiles, int N, int clusters, int k_blocks, int* slices) {
  int best = pairk::BN_MAX, best_s = 1;
  double best_cost = -1;
  for (int bn = pairk::BN_MAX; bn >= 128; bn -= 32) {
    const long tiles = row_tiles * ((N + bn - 1) / bn);
    const long waves = (tiles + clusters - 1) / clusters;
    // One K block of a tile takes (bn + 150) units of about a nanosecond (1000 x 3584 x 8192: 32.5 us a
    // wave at bn = 128, 43.9 at 224).  A cut costs the exchange of the partial sums on top, about 5 us.
    double cost = (double)waves * (bn + 150) * k_blocks;
    int s = 1;
    if (slices) {
      const int cut = (int)std::min<long>(std::min<long>(clusters / tiles, k_blocks / 8), std::min(pairk::MAX_SLICES, bn / 32));
      const double c2 = cut < 2 ? cost : (double)(bn + 150) * ((k_blocks + cut - 1) / cut) + 5000.0;
      if (c2 < cost) {
        cost = c2;
        s = cut;
      }
    }
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = bn;
      best_s = s;
    }
  }
  if (slices) *slices = best_s;
  return best;
}

size_t pair_gemm_ws_bytes(int sms) { return (size_t)sms * pairk::SLOT_FLOATS * sizeof(float); }
size_t pair_gemm_ctr_words(int sms) { return (size_t)2 * sms; }

bool pair_gemm_takes(const PairProblem& p) {
  const int a_inner = p.a_mn ? p.M : p.K, b_inner = p.b_mn ? p.N : p.K;
  return !(((uintptr_t)p.A | (uintptr_t)p.B | (uintptr_t)p.C) & 15) && a_inner % 8 == 0 && b_inner % 8 == 0 && p.N % 8 == 0 && p.groups <= pairk::MAX_GROUPS;
}

namespace pairk {
long row_tiles_of(const PairProblem& d) {   // of 256 rows, over all groups
  const long one = (d.M + TM - 1) / TM;
  return d.mode == kPairPlain ? one : d.mode == kPairGroupedK ? one * d.groups : std::max(1, d.row_tiles_hint);
}
}  // namespace pairk

PairTiling pair_gemm_tiling(const PairProblem& d, int sms, bool may_cut) {
  PairTiling t;
  t.slices = 1;
  may_cut = may_cut && d.mode == kPairPlain && d.epilogue != kPairSwiGLU32;
  t.bn = pair_gemm_pick_bn(pairk::row_tiles_of(d), d.N, std::max(1, sms / 2), (d.K + pairk::BK - 1) / pairk::BK, may_cut ? &t.slices : nullptr);
  if (d.epilogue != kPairStore) t.bn = t.bn > 192 ? 256 : (t.bn > 128 ? 192 : 128);   // gate and up columns in blocks of 32, half a tile each
  if (t.slices > 1) t.slices = std::min(t.slices, (d.epilogue == kPairStore ? t.bn : t.bn / 2) / 32);   // a chunk of the result per slice
  return t;
}

Status launch_pair_gemm(const PairProblem& d, int sms, cudaStream_t stream) {
  pairk::Params p;
  p.C = d.C;
  p.M = d.M;
  p.N = d.N;
  p.K = d.K;
  p.mode = d.mode;
  p.epilogue = d.epilogue;
  p.groups = d.groups;
  p.group_off = d.group_off;
  p.status = d.status;
  p.timeout_ns = d.timeout_ns;
  p.ldc = d.epilogue == kPairStore ? d.N : d.N / 2;
  p.sk_ws = d.sk_ws;
  p.sk_ctr = d.sk_ctr;
  const PairTiling tiling = pair_gemm_tiling(d, sms, d.sk_ws && d.sk_ctr);
  p.bn = tiling.bn;
  p.slices = tiling.slices;
  CUtensorMap ma, mb;
  if (d.a_mn) AMEM_TRY(make_bf16_map(&ma, d.A, d.M, d.K, 1, 64));
  else AMEM_TRY(make_bf16_map(&ma, d.A, d.K, d.M, 1, pairk::HM));
  const uint64_t z = d.mode == kPairGroupedRows ? d.groups : 1;
  if (d.b_mn) AMEM_TRY(make_bf16_map(&mb, d.B, d.N, d.K, z, 64));
  else AMEM_TRY(make_bf16_map(&mb, d.B, d.K, d.N, z, p.bn / 2));
  const int clusters = std::max(1, sms / 2);
  const long tiles = d.mode == kPairGroupedRows ? clusters : pairk::row_tiles_of(d) * ((d.N + p.bn - 1) / p.bn) * p.slices;
  const int grid = 2 * (int)std::min<long>(clusters, std::max<long>(1, tiles));
  if (!d.a_mn && !d.b_mn) return pairk::launch<0, 0>(p, ma, mb, grid, stream);
  if (!d.a_mn) return pairk::launch<0, 1>(p, ma, mb, grid, stream);
  if (d.b_mn) return pairk::launch<1, 1>(p, ma, mb, grid, stream);
  return fail(kInvalidArgument, "pair gemm: A by rows of K with B by rows of N is not built");
}

}  // namespace amem
