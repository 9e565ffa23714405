// tcgen05 GEMM for few rows of activations (decode steps, experts with a handful of tokens).
//
// Such a product takes as long as reading the weights once, so everything here serves that stream:
// the WEIGHTS are the 128-row operand of the tensor core and the tokens its N side (16 .. 128 wide),
// so no MMA row and no byte of shared memory goes to padding tokens; and the K blocks of all weight
// tiles form one sequence that is cut evenly over the SMs, whatever the number of tiles, so every SM
// keeps its whole ring (up to 11 stages, about 190 KB) of weight loads in flight to the end.
// (Several groups: whole tiles, see skinny_gemm_cuts.)
//
// A tile cut by such a boundary is finished by whichever of its CTAs comes last: each parks its fp32
// partial sums (64 KB at most), counts itself in, and the last one adds the parts in order of K -- the
// result does not depend on the order of arrival, and nobody waits for anybody.  With at most half as many tiles
// as SMs and long shares every tile has an owner, which takes the end of its K blocks and LEAD more of them than its helpers take,
// so that their parts have long been parked when it is done: it has added them up by then and does not park its own.
//
// Accumulator rows are output features, so a warp's store of one token covers 32 consecutive features.
// SwiGLU pairs a gate warp with the up warp that holds the same features; they meet in shared memory.
//
// Measured (B200, weights from HBM, us; one-SM kernel -> this one, floor): 16 x 7168 x 8192 37.5 -> 27.8,
// 25.6 with owners (18.0; 2.7 until the first stage has landed), 8 groups of 3072 x 4096
// with 8 rows each and SwiGLU 78.7 (SM pairs) -> 46.6 (30.8).  Stays ahead of the SM pairs up to 64 rows,
// or 96 a group; from there the tokens' share of every stage costs more than the padding it avoids
// (128 rows: 39.1 against 37.2).
//
// TMA loads carry no multicast; every wait is bounded and ends in an error status.
#include <algorithm>

#include "../core/log.h"
#include "coll_device.cuh"
#include "gemm_skinny.h"
#include "pdl.cuh"
#include "sm100_prims.cuh"
#include "smem_limit.h"

namespace amem {
namespace skinnyk {

using namespace sm100;

constexpr int WM = 128, BK = 64;                 // weight rows and K of a stage
constexpr int W_BYTES = WM * BK * 2;
constexpr int MAX_NT = kSkinnyMaxRows, MAX_STAGES = 11;
constexpr int RING_BYTES = 198 * 1024;           // 11 stages of 16 + 2 KB (16 tokens) .. 6 of 32 KB (128 tokens)
constexpr int EPI_WARPS = 4, THREADS = 32 * (2 + EPI_WARPS);
constexpr int MAX_GROUPS = 256;
constexpr int MIN_UNITS = 8;                     // K blocks a CTA takes at least
// K blocks (0.24 us each) that an owner takes longer than its helpers, and the even share from which owners pay.  Back to back,
// even shares / leads of 12 / 24 blocks: 16 x 7168 x 8192 (48 blocks a CTA) 26.2 / 25.4 / 25.0 us, 64 x 7168 x 8192 32.5 / 30.5 / 29.7,
// 16 x 9216 x 8192 31.6 / 30.1 / 29.4; but 16 x 3584 x 8192 (24 blocks) 17.1 / 17.2, 4 x 1024 x 8192 (8) 11.1 / 11.6.
constexpr int LEAD = 24, MIN_OWNED = 32;
constexpr int CH = 16;                           // tokens per epilogue chunk
constexpr size_t SLOT_FLOATS = (size_t)MAX_NT * WM;

struct Params {
  void* C;
  int rows, N, K, ldc, out_cols;
  int nt, stages, epilogue, groups;
  const int* group_off;
  float* ws;          // [CTA][2][token][128]
  uint32_t* ctr;      // [CTA]: parts of the tile whose first K block is this CTA's
  uint32_t* status;
  unsigned long long timeout_ns;
};

struct __align__(8) Ctl {
  uint64_t full[MAX_STAGES], empty[MAX_STAGES];
  uint64_t tfull[2], tempty[2];
  uint32_t tmem_base;
  int abort;
  int last;                         // this CTA came last at its tile
  int off[MAX_GROUPS + 1];
  int first_tile[MAX_GROUPS + 1];
  float up[2][CH][32];              // SwiGLU: the up projection's values, per gate warp
};

// How the K blocks of a product's tiles are shared out: whole tiles; all blocks of all tiles in a row, cut evenly; or the last
// `own` blocks of tile c for CTA c, its owner, and the others of all tiles in a row, cut evenly over the CTAs behind the owners.
enum { WHOLE = 0, EVEN = 1, OWNERS = 2 };
template <int HOW>
struct Share {
  int tiles, nkb, ctas, own;
  __device__ __forceinline__ Share(const Params& p, int tiles_, int grid) {
    tiles = tiles_;
    nkb = (p.K + BK - 1) / BK;
    const long units = (long)tiles * nkb;
    ctas = (int)min((long)grid, max(1L, HOW != WHOLE ? units / MIN_UNITS : (long)tiles));
    own = 0;
    if (HOW == OWNERS) {
      const int lead = min(LEAD, (int)(units / ctas) / 2);
      own = (int)((units - (long)tiles * lead) / ctas) + lead;
    }
  }
  __device__ __forceinline__ int shared() const { return nkb - own; }   // blocks of a tile that its helpers take
  __device__ __forceinline__ long lo(int c) const {
    if (HOW == OWNERS) return (long)(c - tiles) * ((long)tiles * shared()) / (ctas - tiles);
    return HOW == EVEN ? (long)c * ((long)tiles * nkb) / ctas : (long)c * tiles / ctas * nkb;
  }
  __device__ __forceinline__ int holder(long u) const {   // the CTA whose share holds block u of the row
    int c = HOW == OWNERS ? tiles + (int)(u * (ctas - tiles) / ((long)tiles * shared())) : (int)(u * ctas / ((long)tiles * nkb));
    while (lo(c + 1) <= u) ++c;
    while (lo(c) > u) --c;
    return c;
  }
  // This CTA's share, as numbers u0 <= u < u1, and what a run of them from u on is: blocks [kb0, kb1) of tile t.
  __device__ __forceinline__ void mine(int cta, long& u0, long& u1) const {
    const bool busy = tiles > 0 && cta < ctas, owner = HOW == OWNERS && cta < tiles;
    u0 = busy && !owner ? lo(cta) : 0;
    u1 = !busy ? 0 : owner ? own : lo(cta + 1);
  }
  __device__ __forceinline__ void run(int cta, long u, long u1, int& t, int& kb0, int& kb1) const {
    if (HOW == OWNERS && cta < tiles) {
      t = cta;
      kb0 = shared() + (int)u;
      kb1 = nkb;
      return;
    }
    const int per = HOW == OWNERS ? shared() : nkb;
    t = (int)(u / per);
    kb0 = (int)(u - (long)t * per);
    kb1 = (int)min((long)per, kb0 + (u1 - u));
  }
};

struct Tile {
  int group, row0, rows, w_tile;   // token rows of the tile (first in A and C, number), weight row tile
};

__device__ __forceinline__ Tile tile_at(const Params& p, const Ctl* c, int t) {
  int e = 0, hi = p.groups;
  while (hi - e > 1) {
    const int mid = (e + hi) / 2;
    if (c->first_tile[mid] <= t) e = mid;
    else hi = mid;
  }
  const int rows = c->off[e + 1] - c->off[e], blocks = (rows + p.nt - 1) / p.nt, v = t - c->first_tile[e];
  Tile o;
  o.group = e;
  o.w_tile = v / blocks;           // the token blocks of one weight tile are neighbours: W comes from L2 then
  const int b = v - o.w_tile * blocks;
  o.row0 = c->off[e] + b * p.nt;
  o.rows = min(p.nt, rows - b * p.nt);
  return o;
}

__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, unsigned long long timeout_ns, volatile int* abort) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, timeout_ns, abort));
}
__device__ __forceinline__ void tma_load_3d(void* dst, const void* map, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool test_bar(uint64_t* bar, uint32_t parity) {   // does not block
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint32_t count_in(uint32_t* ctr) {
  uint32_t old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(ctr) : "memory");
  return old;
}
// 32 lanes x 16 consecutive fp32 columns
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

// (Kept apart: in one kernel with the others whole tiles took 0.2 us a launch longer.)
template <int HOW>
__global__ void __launch_bounds__(THREADS, 1)
skinny_kernel(const __grid_constant__ Params p, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a) {
  extern __shared__ char smem_raw[];
  char* ring = (char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Ctl* ctl = (Ctl*)(ring + RING_BYTES);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x / 32, 0), lane = threadIdx.x % 32;
  volatile int* abort = &ctl->abort;
  const int nt = p.nt, stages = p.stages, stage_bytes = W_BYTES + nt * BK * 2;
  const uint32_t tmem_cols = (uint32_t)max(32, 2 * nt);
  pdl_launch_dependents();
  const bool swiglu = p.epilogue != kPairStore;
  const int w_tiles = (p.N + WM - 1) / WM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ctl->tfull[b], 1);
      mbar_init(&ctl->tempty[b], EPI_WARPS);
    }
    ctl->abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_a);
  }
  if (warp == 1) {
    tmem_alloc(&ctl->tmem_base, tmem_cols);
    tmem_relinquish();
  }
  pdl_wait();   // from here on: what earlier kernels wrote is read, what they read may be overwritten
  if (warp == 2) {
    if (!p.group_off) {
      if (lane == 0) {
        ctl->off[0] = 0;
        ctl->off[1] = p.rows;
        ctl->first_tile[0] = 0;
        ctl->first_tile[1] = (p.rows + nt - 1) / nt * w_tiles;
      }
    } else {
      int last = 0, carry = 0;
      for (int e0 = 0; e0 <= p.groups; e0 += 32) {   // offsets, made monotonic and kept inside A
        const int e = e0 + lane;
        int v = e <= p.groups ? min(max(p.group_off[e], 0), p.rows) : 0;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
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
        const int n = e < p.groups ? (ctl->off[e + 1] - ctl->off[e] + nt - 1) / nt * w_tiles : 0;
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
  tc_fence_after_sync();
  const uint32_t tmem_base = ctl->tmem_base;

  const Share<HOW> sh(p, ctl->first_tile[p.groups], (int)gridDim.x);
  const int cta = blockIdx.x;
  long u0, u1;
  sh.mine(cta, u0, u1);

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const uint32_t bytes = (uint32_t)stage_bytes;
    for (long u = u0; u < u1 && ok;) {
      int t, kb0, kb1;
      sh.run(cta, u, u1, t, kb0, kb1);
      const Tile tl = tile_at(p, ctl, t);
      for (int kb = kb0; kb < kb1 && ok; ++kb) {
        ok = wait_bar(&ctl->empty[stage], phase ^ 1u, p.timeout_ns, abort);
        if (ok && elect_one()) {
          char* s = ring + (size_t)stage * stage_bytes;
          mbar_expect_tx(&ctl->full[stage], bytes);
          if (p.epilogue == kPairSwiGLUHalves) {   // half a tile of gate rows and the up rows of the same features
            tma_load_3d(s, &map_w, &ctl->full[stage], kb * BK, tl.w_tile * (WM / 2), tl.group);
            tma_load_3d(s + W_BYTES / 2, &map_w, &ctl->full[stage], kb * BK, p.N / 2 + tl.w_tile * (WM / 2), tl.group);
          } else {
            tma_load_3d(s, &map_w, &ctl->full[stage], kb * BK, tl.w_tile * WM, tl.group);
          }
          tma_load_3d(s + W_BYTES, &map_a, &ctl->full[stage], kb * BK, tl.row0, 0);
        }
        __syncwarp();
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      u += kb1 - kb0;
    }
    if (!ok) {
      // gave up: copies that are still in flight land within microseconds; wait for them before leaving
      const unsigned long long t0 = gtimer_ns();
      while (gtimer_ns() - t0 < 2000000ull) {
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t idesc = make_idesc_bf16(WM, nt);
    const uint64_t dw = make_smem_desc_sw128(ring), da = make_smem_desc_sw128(ring + W_BYTES);
    int stage = 0, it = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (long u = u0; u < u1 && ok; ++it) {
      int t, kb0, kb1;
      sh.run(cta, u, u1, t, kb0, kb1);
      const int buf = it & 1;
      ok = wait_bar(&ctl->tempty[buf], (((uint32_t)it >> 1) & 1u) ^ 1u, p.timeout_ns, abort);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t d = tmem_base + (uint32_t)(buf * nt);
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = wait_bar(&ctl->full[stage], phase, p.timeout_ns, abort);
        if (!ok) break;
        tc_fence_after_sync();
        if (elect_one()) {
          const uint64_t at = (uint64_t)((stage * stage_bytes) >> 4);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            tc_mma_f16(d, dw + at + (uint64_t)(kk * 2), da + at + (uint64_t)(kk * 2), idesc, (kb > kb0 || kk) ? 1u : 0u);
          tc_commit(&ctl->empty[stage]);
        }
        __syncwarp();
        if (++stage == stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (ok && elect_one()) tc_commit(&ctl->tfull[buf]);
      __syncwarp();
      u += kb1 - kb0;
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int lg = warp % 4;                       // TMEM lanes [32 * lg, +32)
    // SwiGLU: which warps hold gate rows, and the first feature of this warp's pair inside the tile
    const bool halves = p.epilogue == kPairSwiGLUHalves;
    const bool gate = halves ? lg < 2 : (lg & 1) == 0;
    const int pair = halves ? (lg & 1) : lg / 2;
    int it = 0;
    bool ok = true;
    for (long u = u0; u < u1 && ok; ++it) {
      int t, kb0, kb1;
      sh.run(cta, u, u1, t, kb0, kb1);
      u += kb1 - kb0;
      const Tile tl = tile_at(p, ctl, t);
      const int buf = it & 1;
      const int used = (tl.rows + CH - 1) / CH * CH;   // token columns that matter (rows <= nt, a multiple of CH)
      const int row = lg * 32 + lane;
      // A cut tile's parts, in order of K: those of CTAs c0, c0 + 1, ... and, with owners, the owner's last.
      int c0 = cta, parts = 1;
      const bool is_cut = HOW != WHOLE && (kb0 > 0 || kb1 < sh.nkb);
      if (is_cut) {
        const int per = HOW == OWNERS ? sh.shared() : sh.nkb;
        c0 = sh.holder((long)t * per);
        parts = sh.holder((long)t * per + per - 1) - c0 + 1 + (HOW == OWNERS ? 1 : 0);
      }
      uint32_t* ctr = p.ctr + (HOW == OWNERS ? t : c0);
      auto part_at = [&](int i) {   // (a part that starts its tile lies in its CTA's second slot)
        return p.ws + ((size_t)(HOW == OWNERS && i == parts - 1 ? t : c0 + i) * 2 + (i == 0 ? 1 : 0)) * SLOT_FLOATS + row;
      };
      // the sum of parts [0, n) of tokens [c, c + CH), in order of K; the loads of four parts are in flight together
      auto add_parts = [&](int n, int c, float (&v)[CH]) {
#pragma unroll
        for (int q = 0; q < CH; ++q) v[q] = 0.f;
        for (int i0 = 0; i0 < n; i0 += 4) {
          float x[4][CH];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (i0 + j < n) {
              const float* src = part_at(i0 + j);
#pragma unroll
              for (int q = 0; q < CH; ++q) x[j][q] = __ldcg(src + (size_t)(c + q) * WM);
            }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (i0 + j < n) {
#pragma unroll
              for (int q = 0; q < CH; ++q) v[q] += x[j][q];
            }
        }
      };
      const uint32_t full_parity = ((uint32_t)it >> 1) & 1u;
      bool parked = false;      // the helpers' parts are there before the owner's own
      if (HOW == OWNERS && cta < sh.tiles) {
        if (warp == 2) {
          // until its own is there this warp has nothing else to do than to look for them
          const unsigned long long begin = gtimer_ns();
          for (;;) {
            parked = __shfl_sync(0xffffffffu, lane == 0 ? (int)(ld_acquire(ctr) == (uint32_t)parts - 1u) : 0, 0) != 0;
            if (parked || __any_sync(0xffffffffu, test_bar(&ctl->tfull[buf], full_parity) || *abort || gtimer_ns() - begin > p.timeout_ns)) break;
          }
          if (lane == 0) *(volatile int*)&ctl->last = parked ? 1 : 0;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");
        parked = *(volatile int*)&ctl->last != 0;
      }
      auto accumulated = [&] {
        ok = wait_bar(&ctl->tfull[buf], full_parity, p.timeout_ns, abort);
        if (ok) tc_fence_after_sync();
        return ok;
      };
      if (!(HOW == OWNERS && parked) && !accumulated()) break;
      const uint32_t acc = tmem_base + (uint32_t)(buf * nt) + ((uint32_t)(lg * 32) << 16);
      if (is_cut && !parked) {
        // park this part; whoever comes last adds them all
        float* slot = p.ws + ((size_t)cta * 2 + (kb0 == 0 ? 1 : 0)) * SLOT_FLOATS + row;
        for (int c = 0; c < used; c += CH) {
          uint32_t v[CH];
          tmem_ld_32x16(acc + (uint32_t)c, v);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < CH; ++q) slot[(size_t)(c + q) * WM] = __uint_as_float(v[q]);
        }
        // (one thread orders the parts of all four warps: barrier, release + acquire at the counter, barrier)
        asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");
        if (warp == 2 && lane == 0) {
          const bool last = count_in(ctr) == (uint32_t)parts - 1u;
          if (last) *ctr = 0;
          *(volatile int*)&ctl->last = last ? 1 : 0;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");
        const bool last = *(volatile int*)&ctl->last != 0;
        if (!last) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->tempty[buf]);
          continue;
        }
      }
      const int there = parked ? parts - 1 : parts;   // parts of a cut tile that lie in memory; an owner's is here
      for (int c = 0; c < used; c += CH) {
        float v[CH];
        uint32_t raw[CH];
        if (is_cut) add_parts(there, c, v);
        if (HOW == OWNERS && parked && c == 0) {
          if (!accumulated()) break;
          if (warp == 2 && lane == 0) *ctr = 0;    // (all parts but this one have been counted, and this one never is)
        }
        if (!is_cut || (HOW == OWNERS && parked)) {
          tmem_ld_32x16(acc + (uint32_t)c, raw);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < CH; ++q) v[q] = HOW == OWNERS && is_cut ? v[q] + __uint_as_float(raw[q]) : __uint_as_float(raw[q]);
        }
        int f;
        bool store = true;
        if (swiglu) {
          asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");   // the values of the chunk before have been read
          if (!gate) {
#pragma unroll
            for (int q = 0; q < CH; ++q) ctl->up[pair][q][lane] = v[q];
          }
          asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");
          store = gate;
          if (gate) {
#pragma unroll
            for (int q = 0; q < CH; ++q)   // (zeros of rows that are none would take the quotient's slow path)
              if (c + q < tl.rows) v[q] = v[q] / (1.f + __expf(-v[q])) * ctl->up[pair][q][lane];
          }
          f = tl.w_tile * (WM / 2) + pair * 32 + lane;
        } else {
          f = tl.w_tile * WM + row;
        }
        if (store && f < p.out_cols) {
          __nv_bfloat16* dst = (__nv_bfloat16*)p.C + (size_t)(tl.row0 + c) * p.ldc + f;
#pragma unroll
          for (int q = 0; q < CH; ++q)
            if (c + q < tl.rows) dst[(size_t)q * p.ldc] = __float2bfloat16_rn(v[q]);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->tempty[buf]);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, tmem_cols);
  if (threadIdx.x == 0 && *abort) dev::report_error(p.status, kDevGemmTimeout, 0, 0, (int)blockIdx.x, 0xdead0011u);
}

constexpr size_t kSmemBytes = (size_t)RING_BYTES + sizeof(Ctl) + 1024;
static_assert(kSmemBytes <= 227 * 1024, "ring and control words must fit one SM's shared memory");

}  // namespace skinnyk

size_t skinny_gemm_ws_bytes(int sms) { return (size_t)sms * 2 * skinnyk::SLOT_FLOATS * sizeof(float); }
size_t skinny_gemm_ctr_words(int sms) { return (size_t)sms; }

bool skinny_gemm_takes(const SkinnyProblem& p) {
  return !(((uintptr_t)p.A | (uintptr_t)p.W) & 15) && !((uintptr_t)p.C & 1) && p.K % 8 == 0 && p.groups <= skinnyk::MAX_GROUPS;
}

int skinny_gemm_tokens(const SkinnyProblem& d) {
  // Tokens per tile: all rows of the one group; with several, twice the expected number, so that most
  // groups take one tile (a second one re-reads the weight tile, from L2).
  const int want = d.group_off ? 2 * d.rows_per_group : d.rows;
  return want <= 16 ? 16 : want <= 32 ? 32 : want <= 64 ? 64 : skinnyk::MAX_NT;
}

bool skinny_gemm_cuts(const SkinnyProblem& d, int sms) {
  // Several groups: whole tiles, so that every sum runs over K in one go, as on SM pairs (a caller's guess
  // of the number of rows, which decides between the two kernels, must not show in the result).  One
  // group: cut where that pays.  A stage takes 0.25 us per SM whatever it holds (128 of them 31.4 us with 28 tiles of 128
  // rows, with 56 and with 112 of 64), and no schedule beats reading the weights.  The exchange of a cut takes as much longer
  // than whole tiles take to end as there are tokens' sums to park, and more where shares lie across two tiles than where
  // MIN_UNITS blocks divide a tile.  Back to back, us, whole / cut: 16 x 3584 x 2048 10.5 / 8.0, 16 x 5120 x 2048 (40 tiles: across)
  // 10.5 / 10.8, 16 x 8192 x 3584 16.7 / 17.0, 16 x 7168 x 3584 16.3 / 15.5, 4096 x 4096 17.7 / 12.7; 32 x 4096 x 2048 11.0 / 9.8,
  // 32 x 5120 x 2560 12.9 / 13.8; 64 x 4096 x 2560 13.7 / 17.5, 64 x 7168 x 4096 20.1 / 23.0, 16 x 7168 x 8192 31.7 / 25.0.  Over 864
  // sizes of 1 to 64 tokens the rule loses 25 us in all on the better way of each (one figure of 6.5 for all: 127).
  static const double exchange_us[3][2] = {{3.0, 5.0}, {4.2, 6.4}, {6.5, 8.0}};   // 16, 32, 64 tokens; shares in tiles, across them
  const long w_tiles = (d.N + skinnyk::WM - 1) / skinnyk::WM, nkb = (d.K + skinnyk::BK - 1) / skinnyk::BK;
  const int nt = skinny_gemm_tokens(d);
  const bool across = w_tiles * nkb > (long)skinnyk::MIN_UNITS * sms || nkb % skinnyk::MIN_UNITS != 0;
  const double read_us = (double)d.N * d.K * 2 / 6.5e6;
  const double whole_us = std::max(read_us, (double)((w_tiles + sms - 1) / sms) * nkb * 0.25);
  const double cut_us = std::max(read_us, (double)(w_tiles * nkb) / sms * 0.25) + exchange_us[nt <= 16 ? 0 : nt <= 32 ? 1 : 2][across];
  return !d.group_off && cut_us < whole_us;
}

int skinny_gemm_schedule(const SkinnyProblem& d, int sms, bool workspace) {
  namespace k = skinnyk;
  if (!workspace) return k::WHOLE;
  // Owners need helpers, at least one each (then no helper has parts of more than two tiles), and shares that leave room for a lead.
  const int nt = skinny_gemm_tokens(d);
  const long tiles = (long)((d.rows + nt - 1) / nt) * ((d.N + k::WM - 1) / k::WM), units = tiles * ((d.K + k::BK - 1) / k::BK);
  return !d.group_off && 2 * tiles <= sms && units / sms >= k::MIN_OWNED ? k::OWNERS : k::EVEN;
}

Status launch_skinny_gemm(const SkinnyProblem& d, int sms, cudaStream_t stream) {
  namespace k = skinnyk;
  k::Params p;
  p.C = d.C;
  p.rows = d.rows;
  p.N = d.N;
  p.K = d.K;
  p.out_cols = d.epilogue == kPairStore ? d.N : d.N / 2;
  p.ldc = p.out_cols;
  p.epilogue = d.epilogue;
  p.groups = d.group_off ? d.groups : 1;
  p.group_off = d.group_off;
  p.ws = d.ctr && skinny_gemm_cuts(d, sms) ? d.ws : nullptr;
  p.ctr = d.ctr;
  p.status = d.status;
  p.timeout_ns = d.timeout_ns;
  p.nt = skinny_gemm_tokens(d);
  p.stages = std::min(k::MAX_STAGES, k::RING_BYTES / (k::W_BYTES + p.nt * k::BK * 2));
  CUtensorMap mw, ma;
  AMEM_TRY(make_bf16_map(&mw, d.W, d.K, d.N, p.groups, d.epilogue == kPairSwiGLUHalves ? k::WM / 2 : k::WM));
  AMEM_TRY(make_bf16_map(&ma, d.A, d.K, d.rows, 1, p.nt));
  const int how = skinny_gemm_schedule(d, sms, p.ws != nullptr);
  auto kernel = how == k::WHOLE ? k::skinny_kernel<k::WHOLE> : how == k::OWNERS ? k::skinny_kernel<k::OWNERS> : k::skinny_kernel<k::EVEN>;
  static OncePerDevice raised[3];
  cudaError_t e = allow_smem(raised[how], kernel, k::kSmemBytes);
  if (e != cudaSuccess) return fail(kCudaError, "cudaFuncSetAttribute(%zu bytes of shared memory): %s", k::kSmemBytes, cudaGetErrorString(e));
  e = launch_overlapped(kernel, dim3(sms), dim3(k::THREADS), k::kSmemBytes, stream, p, mw, ma);
  if (e != cudaSuccess) return fail(kCudaError, "skinny gemm launch failed: %s", cudaGetErrorString(e));
  return kSuccess;
}

}  // namespace amem
