// MoE dispatch / combine kernels (sm_100a).  See moe.h for the scheme.  Three launches make a
// dispatch (one, on a single rank with few pairs) -- count (per-segment expert histograms), plan (scan + exchange of the histograms
// between ranks + row offsets), scatter (rows written into the owners' buffers over NVLink) --
// and one launch makes a combine.  Peers are reached with plain 16-byte loads and stores; all
// cross-rank waits go through the bounded block barrier of coll_device.cuh.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "../core/log.h"
#include "coll_device.cuh"
#include "moe.h"
#include "pdl.cuh"
#include "sm100_prims.cuh"
#include "smem_limit.h"

namespace amem {
namespace moek {


constexpr int kThreads = 1024;        // count, plan, scatter: one CTA per SM, 32 warps
constexpr int kCombineThreads = 256;  // up to two CTAs per SM, 128 registers a thread
constexpr int kWarps = kThreads / 32;
// One launch does a whole dispatch of one rank up to this many pairs: every CTA then works out the
// positions of ALL pairs for itself and nothing has to be exchanged.
constexpr int kOneLaunchPairs = 2 * kThreads;

// Segment `seg` of the pairs: whole tokens, so that one CTA holds all choices of a token.
__device__ __forceinline__ void segment_of(const MoeArgs& a, int seg, int segments, int& lo, int& hi) {
  const int per = (a.T + segments - 1) / segments;
  lo = min(a.T, seg * per) * a.k;
  hi = min(a.T, (seg + 1) * per) * a.k;
}
__device__ __forceinline__ int expert_of(const MoeArgs& a, int pair) {   // -1: no such expert, the pair goes nowhere
  const int e = a.topk_idx[pair];
  return e >= 0 && e < a.E ? e : -1;
}

// ---- K1: histogram of expert ids per contiguous segment of (token, choice) pairs
__device__ void count_body(const MoeArgs& a, int seg, int segments) {
  __shared__ int hist[kMoeMaxExperts];
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  int lo, hi;
  segment_of(a, seg, segments, lo, hi);
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const int e = expert_of(a, i);
    if (e >= 0) atomicAdd(&hist[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) a.seg_hist[seg * a.E + e] = hist[e];
}

// Where the rows of every expert lie: offsets of my pairs in the owners' buffers, counts and offsets of
// my own experts.  cnt[s][e] = pairs of rank s for expert e.  Called by a whole CTA.
__device__ void place_experts(const MoeArgs& a, const int (*cnt)[kMoeMaxExperts], int* send_off, bool write_own) {
  const int n = a.coll.nranks, r = a.coll.rank, E = a.E, El = E / n;
  // one warp per owner: a running sum over its experts, 32 at a time
  for (int owner = threadIdx.x / 32; owner < n; owner += blockDim.x / 32) {
    const int lane = threadIdx.x % 32;
    int carry = 0;
    for (int l0 = 0; l0 < El; l0 += 32) {
      const int el = l0 + lane, e = owner * El + el;
      int total = 0, before_me = 0;
      if (el < El)
        for (int s = 0; s < n; ++s) {
          if (s == r) before_me = total;
          total += cnt[s][e];
        }
      int sum = total;
#pragma unroll
      for (int d = 1; d < 32; d *= 2) {
        const int o = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += o;
      }
      const int first = carry + sum - total;
      if (el < El) {
        send_off[e] = first + before_me;
        if (owner == r && write_own) {
          // rows land expert after expert, so the ones beyond the capacity are exactly the tail of
          // this sequence: clamping the running total gives the counts of the rows actually stored
          const int cap = a.capacity_rows, lo = min(first, cap), hi = min(first + total, cap);
          a.expert_counts[el] = hi - lo;
          a.expert_offsets[el] = lo;
          if (el == El - 1) {
            a.expert_offsets[El] = hi;
            if (a.dropped_rows) *a.dropped_rows = max(0, first + total - cap);
          }
        }
      }
      carry += __shfl_sync(0xffffffffu, sum, 31);
    }
  }
}

// ---- K2: one CTA per rank.  Scan the segment histograms, all-gather the per-expert totals
// through the control blocks, derive where my rows start in every owner's buffer.
__device__ void plan_body(const MoeArgs& a, int segments, int* s_abort) {
  __shared__ int cnt[kMaxRanks][kMoeMaxExperts];
  const int n = a.coll.nranks, r = a.coll.rank, E = a.E;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nwarps = blockDim.x / 32;
  dev::Proto p;
  dev::proto_begin(p, a.coll, 0, 1, s_abort);
  // A warp takes an expert, a lane four neighbouring segments: the loads of an expert are in flight
  // together (one thread per expert walked 128 dependent steps: 41 us for 64 experts, now 8).
  for (int e = warp; e < E; e += nwarps) {
    int carry = 0;
    for (int s0 = 0; s0 < segments; s0 += 128) {
      int h[4], sum = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int s = s0 + lane * 4 + j;
        h[j] = s < segments ? a.seg_hist[s * E + e] : 0;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) sum += h[j];
      int scan = sum;
#pragma unroll
      for (int d = 1; d < 32; d *= 2) {
        const int o = __shfl_up_sync(0xffffffffu, scan, d);
        if (lane >= d) scan += o;
      }
      int run = carry + scan - sum;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int s = s0 + lane * 4 + j;
        if (s < segments) a.seg_base[s * E + e] = run;
        run += h[j];
      }
      carry += __shfl_sync(0xffffffffu, scan, 31);
    }
    if (lane == 0) cnt[r][e] = carry;
  }
  if (n > 1) {
    // peers may still read the totals of the previous dispatch: they signal this barrier only
    // after they have left it
    dev::block_barrier(p);
    for (int e = threadIdx.x; e < E; e += blockDim.x)
      for (int q = 0; q < n; ++q) a.coll.ctrl[q]->xchg[r][e] = (uint32_t)cnt[r][e];
    dev::block_barrier(p);
    for (int i = threadIdx.x; i < n * E; i += blockDim.x) {
      int s = i / E, e = i % E;
      cnt[s][e] = (int)dev::ld_volatile(&a.coll.ctrl[r]->xchg[s][e]);
    }
  }
  __syncthreads();
  place_experts(a, cnt, a.send_off, true);
  dev::proto_end(p);
}

// Positions of up to blockDim.x pairs at once: thread i holds expert e (-1: none) of pair i of the chunk;
// run[e] = rows of expert e placed before the chunk, updated.  Rows keep pair order inside an expert.
// whist: [warps][E | 1] scratch.  Called by a whole CTA.
__device__ int chunk_positions(int e, int E, int* run, int* whist) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nwarps = blockDim.x / 32;
  const int stride = E | 1;   // odd: a column of the table lies in 32 banks
  for (int i = threadIdx.x; i < nwarps * stride; i += blockDim.x) whist[i] = 0;
  __syncthreads();
  const unsigned same = __match_any_sync(0xffffffffu, e);
  const int before = __popc(same & ((1u << lane) - 1u));
  if (e >= 0 && before == 0) whist[warp * stride + e] = __popc(same);
  __syncthreads();
  for (int x = warp; x < E; x += nwarps) {   // exclusive sums over the warps: a warp per expert (at most 32 warps)
    const int c = lane < nwarps ? whist[lane * stride + x] : 0, start = run[x];
    int sum = c;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
      const int o = __shfl_up_sync(0xffffffffu, sum, d);
      if (lane >= d) sum += o;
    }
    if (lane < nwarps) whist[lane * stride + x] = start + sum - c;
    if (lane == 31) run[x] = start + sum;
  }
  __syncthreads();
  return e >= 0 ? whist[warp * stride + e] + before : -1;
}

// Copies the rows of the chunk's tokens to the positions of their pairs: a warp takes 4 KB of a token's
// row at a time, reads it once and stores it to every choice.  c_pos / c_exp: the chunk's pairs.
__device__ void copy_rows(const MoeArgs& a, int base, int count, const int* c_pos, const int* c_exp, int first_warp, int all_warps) {
  const int lane = threadIdx.x % 32, El = a.E / a.coll.nranks;
  const size_t row_bytes = (size_t)a.d * 2;
  const int nvec = (int)(row_bytes / 16), parts = (nvec + 255) / 256;
  const int t0 = base / a.k, t1 = (base + count - 1) / a.k;
  for (int item = first_warp; item < (t1 - t0 + 1) * parts; item += all_warps) {
    const int t = t0 + item / parts, v0 = (item % parts) * 256 + lane;
    const uint4* src = (const uint4*)((const char*)a.x + (size_t)t * row_bytes);
    uint4 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (v0 + j * 32 < nvec) v[j] = src[v0 + j * 32];
    const int j0 = max(t * a.k, base) - base, j1 = min((t + 1) * a.k, base + count) - base;
    for (int c = j0; c < j1; ++c) {
      const int pos = c_pos[c];
      if (pos < 0) continue;
      uint4* dst = (uint4*)(a.recv[c_exp[c] / El] + (size_t)pos * row_bytes);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (v0 + j * 32 < nvec) dst[v0 + j * 32] = v[j];
    }
  }
}

// The pairs of a segment to their places; run[e]: where this segment's rows of expert e begin.  Bound by
// the rows' stores (16384 tokens x 8 choices x 8 KB: a row read per pair and 8 warps an SM 467 us; each
// token read once by 32 warps an SM, with the counting 238; 185 are the rows' bytes).
__device__ void scatter_segment(const MoeArgs& a, int seg, int segments, int* run, int* whist) {
  __shared__ int c_pos[kThreads];
  __shared__ int c_exp[kThreads];
  int lo, hi;
  segment_of(a, seg, segments, lo, hi);
  for (int base = lo; base < hi; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int e = i < hi ? expert_of(a, i) : -1;
    int pos = chunk_positions(e, a.E, run, whist);
    if (pos >= a.capacity_rows) pos = -1;  // no room at the owner: not sent (place_experts counted it)
    if (i < hi) a.send_pos[i] = pos;
    c_pos[threadIdx.x] = pos;
    c_exp[threadIdx.x] = e;
    __syncthreads();
    copy_rows(a, base, min((int)blockDim.x, hi - base), c_pos, c_exp, threadIdx.x / 32, blockDim.x / 32);
    __syncthreads();
  }
}

// ---- K3: every pair's row goes to its final place in the owner's receive buffer.
__device__ void scatter_body(const MoeArgs& a, int seg, int segments, int* s_abort) {
  extern __shared__ int whist[];
  __shared__ int run[kMoeMaxExperts];
  dev::Proto p;
  dev::proto_begin(p, a.coll, seg, segments, s_abort);
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) run[e] = a.send_off[e] + a.seg_base[seg * a.E + e];
  scatter_segment(a, seg, segments, run, whist);
  // my rows are out; when this barrier passes on every block of a rank, every rank's rows for
  // it have landed (all ranks run the same number of blocks)
  dev::block_barrier(p);
  dev::proto_end(p);
}

// ---- K2 and K3 of a communicator of one rank: every CTA sums the histograms itself (a few hundred
// bytes per expert, out of L2), so no single CTA's scan stands between counting and copying (41 us of
// the 512 for 64 experts).  CTA 0 writes the tables.
__device__ void place_and_scatter_body(const MoeArgs& a, int seg, int segments) {
  extern __shared__ int whist[];
  __shared__ int run[kMoeMaxExperts];
  __shared__ int before[kMoeMaxExperts];
  __shared__ int cnt[1][kMoeMaxExperts];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nwarps = blockDim.x / 32;
  for (int e = warp; e < a.E; e += nwarps) {
    int total = 0, mine = 0;
    for (int s = lane; s < segments; s += 32) {
      const int h = a.seg_hist[s * a.E + e];
      total += h;
      if (s < seg) mine += h;
    }
    total = __reduce_add_sync(0xffffffffu, total);
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) {
      cnt[0][e] = total;
      before[e] = mine;
    }
  }
  __syncthreads();
  place_experts(a, cnt, run, seg == 0);
  __syncthreads();
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) run[e] += before[e];
  __syncthreads();
  scatter_segment(a, seg, segments, run, whist);
}

// ---- the whole dispatch of a communicator of one rank, for few pairs (see kOneLaunchPairs).  CTA 0
// writes the tables, every CTA copies its share of the rows.
__device__ void small_dispatch_body(const MoeArgs& a, int cta, int nctas) {
  extern __shared__ int whist[];
  __shared__ int run[kMoeMaxExperts];
  __shared__ int off[kMoeMaxExperts];
  __shared__ int cnt[1][kMoeMaxExperts];
  __shared__ int c_pos[kThreads];
  __shared__ int c_exp[kThreads];
  const int P = a.T * a.k;
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) cnt[0][e] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    const int e = expert_of(a, i);
    if (e >= 0) atomicAdd(&cnt[0][e], 1);
  }
  __syncthreads();
  place_experts(a, cnt, off, cta == 0);
  __syncthreads();
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) run[e] = off[e];
  __syncthreads();
  for (int base = 0; base < P; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int e = i < P ? expert_of(a, i) : -1;
    int pos = chunk_positions(e, a.E, run, whist);
    if (pos >= a.capacity_rows) pos = -1;
    if (i < P && cta == 0) a.send_pos[i] = pos;
    c_pos[threadIdx.x] = pos;
    c_exp[threadIdx.x] = e;
    __syncthreads();
    copy_rows(a, base, min((int)blockDim.x, P - base), c_pos, c_exp, (threadIdx.x / 32) * nctas + cta, nctas * (blockDim.x / 32));
    __syncthreads();
  }
}

// ---- combine: out[t] = sum_j w[t,j] * y_owner(t,j)[row(t,j)].  A warp takes VPL x 512 bytes of a token's
// result at a time, KC choices at once, so that 8 to 16 loads are in flight per lane whatever their number (16384 x 8 rows of 8 KB: a token per warp and one vector at a time 434 us, so 227, 185 being the
// rows' bytes; 8192 x 2 rows 96 and 42).
template <int KC, int VPL>
__device__ void combine_items(const MoeArgs& a, int cta, int nctas) {
  const bool one = a.coll.nranks == 1;
  const int El = a.E / a.coll.nranks;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nwarps = blockDim.x / 32;
  const int nvec = a.d / 8, parts = (nvec + 32 * VPL - 1) / (32 * VPL);
  uint4* out = (uint4*)a.out;
  for (long item = (long)warp * nctas + cta; item < (long)a.T * parts; item += (long)nctas * nwarps) {
    const int t = (int)(item / parts), v0 = (int)(item - (long)t * parts) * 32 * VPL + lane;
    float acc[VPL][8];
#pragma unroll
    for (int u = 0; u < VPL; ++u)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[u][q] = 0.f;
    for (int j0 = 0; j0 < a.k; j0 += KC) {
      uint4 raw[KC][VPL];
      float w[KC];
      if (KC < 8) {
        // lane jj looks up choice j0 + jj, the others get it from there
        float my_w = 0.f;
        const uint4* my_row = nullptr;
        if (lane < KC && j0 + lane < a.k) {
          const size_t at = (size_t)t * a.k + j0 + lane;
          const int pos = a.send_pos[at];
          if (pos >= 0 && pos < a.capacity_rows) {
            my_w = a.topk_w[at];
            my_row = (const uint4*)(a.ybuf[one ? 0 : a.topk_idx[at] / El] + (size_t)pos * a.d * 2);
          }
        }
#pragma unroll
        for (int jj = 0; jj < KC; ++jj) {
          const uint4* row = (const uint4*)__shfl_sync(0xffffffffu, (unsigned long long)my_row, jj);
          w[jj] = __shfl_sync(0xffffffffu, my_w, jj);
#pragma unroll
          for (int u = 0; u < VPL; ++u) raw[jj][u] = row && v0 + u * 32 < nvec ? row[v0 + u * 32] : make_uint4(0, 0, 0, 0);
        }
      } else {
        // (with eight choices every lane looks all of them up: shared row pointers need more registers
        // than two CTAs an SM leave, 309 us instead of 227 for 16384 x 8 rows)
#pragma unroll
        for (int jj = 0; jj < KC; ++jj) {
          const int j = j0 + jj;
          w[jj] = 0.f;
#pragma unroll
          for (int u = 0; u < VPL; ++u) raw[jj][u] = make_uint4(0, 0, 0, 0);
          if (j < a.k) {
            const int pos = a.send_pos[(size_t)t * a.k + j];
            if (pos >= 0 && pos < a.capacity_rows) {
              const int owner = a.topk_idx[(size_t)t * a.k + j] / El;
              w[jj] = a.topk_w[(size_t)t * a.k + j];
              const uint4* row = (const uint4*)(a.ybuf[owner] + (size_t)pos * a.d * 2);
#pragma unroll
              for (int u = 0; u < VPL; ++u)
                if (v0 + u * 32 < nvec) raw[jj][u] = row[v0 + u * 32];
            }
          }
        }
      }
#pragma unroll
      for (int jj = 0; jj < KC; ++jj)
#pragma unroll
        for (int u = 0; u < VPL; ++u) {
          const __nv_bfloat16* h = (const __nv_bfloat16*)&raw[jj][u];
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[u][q] = fmaf(w[jj], __bfloat162float(h[q]), acc[u][q]);
        }
    }
#pragma unroll
    for (int u = 0; u < VPL; ++u) {
      if (v0 + u * 32 < nvec) {
        alignas(16) __nv_bfloat16 res[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) res[q] = __float2bfloat16_rn(acc[u][q]);
        out[(size_t)t * nvec + v0 + u * 32] = *(const uint4*)res;
      }
    }
  }
}
template <int KC, int VPL>
__device__ void combine_body(const MoeArgs& a, int cta, int nctas, int* s_abort) {
  dev::Proto p;
  dev::proto_begin(p, a.coll, cta, nctas, s_abort);
  if (a.coll.nranks > 1) dev::block_barrier(p);  // the expert outputs of every rank are complete
  combine_items<KC, VPL>(a, cta, nctas);
  // nobody may overwrite its expert outputs while a peer still reads them
  if (a.coll.nranks > 1) dev::block_barrier(p);
  dev::proto_end(p);
}

// ---- combine of one rank with many choices and long rows: the bulk-copy engine gathers the rows of one token after the
// other (eight choices and a piece of the row a stage) into a ring that never runs dry, and eight warps add them up; the
// sums are those of combine_items, choice after choice.  A warp that loads its own rows has none in flight while it looks
// up the next ones and stores: 16384 x 8 rows of 8 KB 233 us, so 204 (185 are the bytes).  With two choices a stage is too
// short to pay for its barriers: 8192 x 2 rows 38 us against 49.
constexpr int kStreamWarps = 8, kStreamThreads = 32 * (kStreamWarps + 1), kStreamRows = 8, kStreamStages = 16;
constexpr uint32_t kStreamRing = 192 * 1024, kStreamPiece = 8192;   // bytes of the ring; of a row at a time, at most
// A stage takes the same time for pieces of 4 KB as for 6 (16384 x 8 rows in 151 - 184 us for 4 to 6 KB, and 195 for 7, 201 for 8), so
// short pieces are left to combine_items (129 - 182, 209, 240): rows of less than 6 KB but where there are so few of them that
// looking them up in time is what counts (of 4 KB, stream / items: 4096 x 5 rows 37 / 41, 4096 x 6 41 / 43, 4096 x 8 45 / 45, 8192 x 8
// 82 / 74), and rows that come to short pieces (of 8208 bytes: 520 x 8 23 / 19, 8192 x 8 191 / 139; of 16400: 8192 x 8 277 / 248).
// At 6 KB: 16384 x 5 141 / 166, x 6 156 / 172, x 8 184 / 182, 4096 x 12 76 / 88.  Five choices of 8 KB: 150 / 221; four: not
// taken, a stage of half the rows.  520 x 8 rows of 8 KB: 18.5 either way.
constexpr long kStreamMinRows = 4096, kStreamFewRows = 24576;
constexpr uint32_t kStreamShortRow = 4096, kStreamShortPiece = 6144;
// Equal pieces of a row, multiples of 16 bytes.
__host__ __device__ inline uint32_t stream_piece(size_t row_bytes) {
  const size_t parts = (row_bytes + kStreamPiece - 1) / kStreamPiece;
  return (uint32_t)((row_bytes / 16 + parts - 1) / parts * 16);
}
struct StreamCtl {
  uint64_t full[kStreamStages], empty[kStreamStages];
  float w[kStreamStages][kStreamRows];
  uint32_t kept[kStreamStages];   // bit r: row r of the stage is there
  int abort;
};
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sm100::smem_u32(dst)), "l"(src), "r"(bytes),
               "r"(sm100::smem_u32(bar)) : "memory");
}
__global__ void __launch_bounds__(kStreamThreads, 1) combine_stream_kernel(const __grid_constant__ MoeArgs a, int stages) {
  extern __shared__ __align__(128) char ring[];   // [stages][min(k, kStreamRows)][piece]
  __shared__ StreamCtl ctl;
  pdl_launch_dependents();
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x / 32, 0), lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      sm100::mbar_init(&ctl.full[s], 1);
      sm100::mbar_init(&ctl.empty[s], kStreamWarps);
    }
    ctl.abort = 0;
    sm100::mbar_fence_init();
  }
  __syncthreads();
  pdl_wait();
  const size_t row_bytes = (size_t)a.d * 2;
  const uint32_t piece = stream_piece(row_bytes);
  const int kc = min(a.k, kStreamRows), passes = (a.k + kStreamRows - 1) / kStreamRows, parts = (int)((row_bytes + piece - 1) / piece);
  const int items = a.T * parts;     // (the launch keeps it below 2^30)
  auto length = [&](int part) { return (uint32_t)min((size_t)piece, row_bytes - (size_t)part * piece); };
  int stage = 0;
  uint32_t phase = 0;
  auto next = [&] {
    if (++stage == stages) {
      stage = 0;
      phase ^= 1u;
    }
  };
  bool ok = true;
  if (warp == kStreamWarps) {
    // lane r looks up and fetches row r of a stage; what it looks up for the next stage is on its way meanwhile
    int pos_next = -1;
    float w_next = 0.f;
    auto look_up = [&](int item, int pass) {
      const int j = pass * kStreamRows + lane;
      pos_next = -1;
      w_next = 0.f;
      if (lane < kc && item < items && j < a.k) {
        const size_t at = (size_t)(item / parts) * a.k + j;
        pos_next = a.send_pos[at];
        w_next = a.topk_w[at];
      }
    };
    look_up(blockIdx.x, 0);
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      const int part = item % parts;
      const uint32_t len = length(part);
      for (int pass = 0; pass < passes; ++pass) {
        const int pos = pos_next;
        const float w = w_next;
        if (pass + 1 < passes) look_up(item, pass + 1);
        else look_up(item + gridDim.x, 0);
        const bool row = pos >= 0 && pos < a.capacity_rows;
        const uint32_t kept = __ballot_sync(0xffffffffu, row);
        ok = __all_sync(0xffffffffu, sm100::mbar_wait(&ctl.empty[stage], phase ^ 1u, a.coll.timeout_ns, &ctl.abort));
        if (!ok) break;
        if (lane < kc) ctl.w[stage][lane] = w;
        if (lane == 0) ctl.kept[stage] = kept;
        __syncwarp();
        if (lane == 0) sm100::mbar_expect_tx(&ctl.full[stage], (uint32_t)__popc(kept) * len);
        __syncwarp();
        if (row) bulk_g2s(ring + ((size_t)stage * kc + lane) * piece, a.ybuf[0] + (size_t)pos * row_bytes + (size_t)part * piece, len, &ctl.full[stage]);
        next();
      }
    }
    if (!ok) {
      // gave up: copies that are still in flight land within microseconds; wait for them before leaving
      const unsigned long long begin = sm100::gtimer_ns();
      while (sm100::gtimer_ns() - begin < 2000000ull) {
      }
    }
  } else {
    constexpr int VPL = kStreamPiece / 16 / (32 * kStreamWarps);
    for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
      const int part = item % parts;
      const uint32_t len = length(part);
      float acc[VPL][8];
#pragma unroll
      for (int u = 0; u < VPL; ++u)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[u][q] = 0.f;
      for (int pass = 0; pass < passes; ++pass) {
        ok = __all_sync(0xffffffffu, sm100::mbar_wait(&ctl.full[stage], phase, a.coll.timeout_ns, &ctl.abort));
        if (!ok) break;
        const uint32_t kept = ctl.kept[stage];
        const char* rows = ring + (size_t)stage * kc * piece;
#pragma unroll
        for (int j = 0; j < kStreamRows; ++j)
          if (kept >> j & 1u) {
            const float w = ctl.w[stage][j];
#pragma unroll
            for (int u = 0; u < VPL; ++u) {
              const uint32_t v = (threadIdx.x + u * 32 * kStreamWarps) * 16;
              if (v < len) {
                const uint4 raw = *(const uint4*)(rows + (size_t)j * piece + v);
                const __nv_bfloat16* h = (const __nv_bfloat16*)&raw;
#pragma unroll
                for (int q = 0; q < 8; ++q) acc[u][q] = fmaf(w, __bfloat162float(h[q]), acc[u][q]);
              }
            }
          }
        __syncwarp();
        if (lane == 0) sm100::mbar_arrive(&ctl.empty[stage]);
        next();
      }
      if (!ok) break;
      char* out = (char*)a.out + (size_t)(item / parts) * row_bytes + (size_t)part * piece;
#pragma unroll
      for (int u = 0; u < VPL; ++u) {
        const uint32_t v = (threadIdx.x + u * 32 * kStreamWarps) * 16;
        if (v < len) {
          alignas(16) __nv_bfloat16 res[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) res[q] = __float2bfloat16_rn(acc[u][q]);
          *(uint4*)(out + v) = *(const uint4*)res;
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && *(volatile int*)&ctl.abort) dev::report_error(a.coll.status, kDevBarrierTimeout, a.coll.rank, a.coll.rank, (int)blockIdx.x, 0xdead0021u);
}

// ---- the combine's backward on one rank: for every kept choice j of token t, with row p = row(t, j),
// g_w[t, j] = <g_out[t], y[p]> and g_y[p] = w[t, j] * g_out[t].  A CTA per token: the token's gradient comes
// from HBM once, each expert row is read and each gradient row written once (as a gather of the outputs, a
// product, a sum, a scaled copy and a second dispatch: 0.5 ms for 4096 x 2 rows of 8 KB; 27.5 us so,
// 25 are the bytes).
constexpr int kGradThreads = 128;
constexpr int kGradAhead = 4;   // vectors of either row that a thread loads ahead of its stores: all of them up to d = 4096
__global__ void __launch_bounds__(kGradThreads) combine_grad_kernel(const char* g_out, const char* y, const float* w, const int* send_pos, char* g_y,
                                                                    float* g_w, int rows, int T, int k, int d) {
  __shared__ float part[kGradThreads / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nvec = d / 8;
  const size_t row_bytes = (size_t)d * 2;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    const uint4* g = (const uint4*)(g_out + (size_t)t * row_bytes);
    for (int j = 0; j < k; ++j) {
      const size_t at = (size_t)t * k + j;
      const int pos = send_pos[at];   // the same for the whole CTA
      if (pos < 0 || pos >= rows) {
        if (threadIdx.x == 0) g_w[at] = 0.f;
        continue;
      }
      const float scale = w[at];
      const uint4* src = (const uint4*)(y + (size_t)pos * row_bytes);
      uint4* dst = (uint4*)(g_y + (size_t)pos * row_bytes);
      float dot = 0.f;
      for (int v0 = threadIdx.x; v0 < nvec; v0 += kGradAhead * kGradThreads) {
        uint4 gr[kGradAhead], yr[kGradAhead];
#pragma unroll
        for (int i = 0; i < kGradAhead; ++i)
          if (v0 + i * kGradThreads < nvec) {
            gr[i] = g[v0 + i * kGradThreads];
            yr[i] = src[v0 + i * kGradThreads];
          }
#pragma unroll
        for (int i = 0; i < kGradAhead; ++i)
          if (v0 + i * kGradThreads < nvec) {
            const __nv_bfloat16 *gh = (const __nv_bfloat16*)&gr[i], *yh = (const __nv_bfloat16*)&yr[i];
            alignas(16) __nv_bfloat16 res[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const float gf = __bfloat162float(gh[q]);
              dot = fmaf(gf, __bfloat162float(yh[q]), dot);
              res[q] = __float2bfloat16_rn(gf * scale);
            }
            dst[v0 + i * kGradThreads] = *(const uint4*)res;
          }
      }
#pragma unroll
      for (int o = 16; o > 0; o /= 2) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      if (lane == 0) part[warp] = dot;
      __syncthreads();
      if (threadIdx.x == 0) {
        float sum = 0.f;
        for (int i = 0; i < kGradThreads / 32; ++i) sum += part[i];
        g_w[at] = sum;
      }
      __syncthreads();
    }
  }
}

// ---- the input's gradient of routing and dispatch together, on one rank: g_x[t] = sum over the choices of the row's gradient
// and of the logit's gradient times the expert's router row.  Warps take pieces of a token as in combine_items, two choices'
// rows and router rows in flight; the router's come out of L2.  4096 x 2 rows of 8 KB: as a combine with unit weights, a product
// and an addition 47 us, so 22.8 (15 are the bytes; cold, under ncu).
constexpr int kInputVPL = 4;
__global__ void __launch_bounds__(kCombineThreads, 2) input_grad_kernel(const char* g_rows, const int* send_pos, const int* idx, const __nv_bfloat16* g_logits,
                                                                        const char* router, char* g_x, int rows, int T, int k, int d, int E) {
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nwarps = blockDim.x / 32, nvec = d / 8, parts = (nvec + 32 * kInputVPL - 1) / (32 * kInputVPL);
  const size_t row_bytes = (size_t)d * 2;
  for (long item = (long)warp * gridDim.x + blockIdx.x; item < (long)T * parts; item += (long)gridDim.x * nwarps) {
    const int t = (int)(item / parts), v0 = (int)(item - (long)t * parts) * 32 * kInputVPL + lane;
    float acc[kInputVPL][8];
#pragma unroll
    for (int u = 0; u < kInputVPL; ++u)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[u][q] = 0.f;
    for (int j0 = 0; j0 < k; j0 += 32) {
      // lane j looks up choice j0 + j, the others get it from there
      int pos = -1, e = 0;
      float g = 0.f;
      if (j0 + lane < k) {
        const size_t at = (size_t)t * k + j0 + lane;
        pos = send_pos[at];
        e = idx[at];
        if (e >= 0 && e < E) g = __bfloat162float(g_logits[(size_t)t * E + e]);
        else e = -1;
      }
#pragma unroll 2
      for (int j = 0; j < min(32, k - j0); ++j) {
        const int p = __shfl_sync(0xffffffffu, pos, j), ex = __shfl_sync(0xffffffffu, e, j);
        const float gl = __shfl_sync(0xffffffffu, g, j);
        const bool kept = p >= 0 && p < rows;
        const uint4 *row = (const uint4*)(g_rows + (size_t)max(p, 0) * row_bytes), *of_expert = (const uint4*)(router + (size_t)max(ex, 0) * row_bytes);
        uint4 a[kInputVPL], b[kInputVPL];
#pragma unroll
        for (int u = 0; u < kInputVPL; ++u) {
          const int v = v0 + u * 32;
          a[u] = kept && v < nvec ? row[v] : make_uint4(0, 0, 0, 0);
          b[u] = ex >= 0 && v < nvec ? of_expert[v] : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < kInputVPL; ++u) {
          const __nv_bfloat16 *ah = (const __nv_bfloat16*)&a[u], *bh = (const __nv_bfloat16*)&b[u];
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[u][q] = fmaf(gl, __bfloat162float(bh[q]), acc[u][q] + __bfloat162float(ah[q]));
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kInputVPL; ++u)
      if (v0 + u * 32 < nvec) {
        alignas(16) __nv_bfloat16 res[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) res[q] = __float2bfloat16_rn(acc[u][q]);
        ((uint4*)(g_x + (size_t)t * row_bytes))[v0 + u * 32] = *(const uint4*)res;
      }
  }
}

// ---- kernels: one rank per launch, and all ranks of an emulated communicator per launch
__global__ void __launch_bounds__(kThreads) count_kernel(const __grid_constant__ MoeArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  count_body(a, blockIdx.x, gridDim.x);
}
// (plan and scatter run between ranks only and wait for peers: whatever follows them keeps its turn)
__global__ void __launch_bounds__(kThreads) plan_kernel(const __grid_constant__ MoeArgs a, int segments) {
  __shared__ int s_abort;
  plan_body(a, segments, &s_abort);
}
__global__ void __launch_bounds__(kThreads) scatter_kernel(const __grid_constant__ MoeArgs a) {
  __shared__ int s_abort;
  scatter_body(a, blockIdx.x, gridDim.x, &s_abort);
}
__global__ void __launch_bounds__(kThreads) place_and_scatter_kernel(const __grid_constant__ MoeArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  place_and_scatter_body(a, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(kThreads) small_dispatch_kernel(const __grid_constant__ MoeArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  small_dispatch_body(a, blockIdx.x, gridDim.x);
}
template <int KC, int VPL>
__global__ void __launch_bounds__(kCombineThreads, 2) combine_kernel(const __grid_constant__ MoeArgs a) {
  __shared__ int s_abort;
  if (a.coll.nranks == 1) {
    pdl_launch_dependents();
    pdl_wait();
  }
  combine_body<KC, VPL>(a, blockIdx.x, gridDim.x, &s_abort);
}
__global__ void __launch_bounds__(kThreads) count_kernel_emu(const MoeArgs* __restrict__ all) { count_body(all[blockIdx.y], blockIdx.x, gridDim.x); }
__global__ void __launch_bounds__(kThreads) plan_kernel_emu(const MoeArgs* __restrict__ all, int segments) {
  __shared__ int s_abort;
  plan_body(all[blockIdx.y], segments, &s_abort);
}
__global__ void __launch_bounds__(kThreads) scatter_kernel_emu(const MoeArgs* __restrict__ all) {
  __shared__ int s_abort;
  scatter_body(all[blockIdx.y], blockIdx.x, gridDim.x, &s_abort);
}
__global__ void __launch_bounds__(kCombineThreads, 2) combine_kernel_emu(const MoeArgs* __restrict__ all) {
  __shared__ int s_abort;
  combine_body<8, 2>(all[blockIdx.y], blockIdx.x, gridDim.x, &s_abort);
}

// Per-warp histograms of chunk_positions: at most 33 KB.
size_t whist_bytes(int E) { return (size_t)kWarps * (E | 1) * sizeof(int); }

}  // namespace moek

static Status launched(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(kCudaError, "%s launch failed: %s", what, cudaGetErrorString(e));
  }
  return kSuccess;
}

// One rank: launches overlap their predecessor's end, and their successor theirs.  With peers they are
// ordinary launches and let nobody in early: those kernels wait for the other GPUs', and a successor parked
// on the SMs meanwhile would keep out the kernel of another stream that a peer's progress may depend on.
template <typename... P, typename... A>
static cudaError_t launch(void (*kernel)(P...), const MoeArgs& a, int grid, int threads, size_t smem, cudaStream_t stream, const A&... args) {
  if (a.coll.nranks == 1) return launch_overlapped(kernel, dim3(grid), dim3(threads), smem, stream, args...);
  kernel<<<grid, threads, smem, stream>>>(args...);
  return cudaGetLastError();
}

Status launch_moe_dispatch(const MoeArgs& a, cudaStream_t stream) {
  const size_t smem = moek::whist_bytes(a.E);
  const long pairs = (long)a.T * a.k;
  if (a.coll.nranks == 1 && pairs <= moek::kOneLaunchPairs) {
    // as many CTAs as there are 4 KB pieces for their warps (the positions of all pairs are worked out in each)
    const long pieces = (long)a.T * ((a.d / 8 + 255) / 256);
    const int grid = (int)std::max<long>(1, std::min<long>(kMoeSegments, (pieces + 7) / 8));
    return launched(launch(moek::small_dispatch_kernel, a, grid, moek::kThreads, smem, stream, a), "moe dispatch");
  }
  AMEM_TRY(launched(launch(moek::count_kernel, a, kMoeSegments, moek::kThreads, 0, stream, a), "moe count"));
  if (a.coll.nranks == 1) return launched(launch(moek::place_and_scatter_kernel, a, kMoeSegments, moek::kThreads, smem, stream, a), "moe scatter");
  AMEM_TRY(launched(launch(moek::plan_kernel, a, 1, moek::kThreads, 0, stream, a, kMoeSegments), "moe plan"));
  return launched(launch(moek::scatter_kernel, a, kMoeSegments, moek::kThreads, smem, stream, a), "moe scatter");
}

bool moe_combine_streams(int T, int k, int d) {
  using namespace moek;
  const size_t row = (size_t)d * 2, parts = (row + kStreamPiece - 1) / kStreamPiece;
  const long rows = (long)T * k;
  if (k <= 4 || row < kStreamShortRow || rows < kStreamMinRows || (long)T * (long)parts >= 0x40000000L) return false;
  return stream_piece(row) >= kStreamShortPiece || (parts == 1 && rows <= kStreamFewRows);
}

Status launch_moe_combine(const MoeArgs& a, cudaStream_t stream) {
  if (a.coll.nranks == 1 && moe_combine_streams(a.T, a.k, a.d)) {
    using namespace moek;
    const size_t row = (size_t)a.d * 2;
    const long items = (long)a.T * (long)((row + kStreamPiece - 1) / kStreamPiece);
    const uint32_t stage = (uint32_t)std::min(a.k, kStreamRows) * stream_piece(row);
    const int stages = (int)std::min<uint32_t>(kStreamStages, kStreamRing / stage);
    static OncePerDevice raised;
    const cudaError_t ready = allow_smem(raised, combine_stream_kernel, kStreamRing);
    if (ready != cudaSuccess) return launched(ready, "moe combine (shared memory)");
    return launched(launch(combine_stream_kernel, a, (int)std::min<long>(items, kMoeSegments), kStreamThreads, stages * stage, stream, a, stages), "moe combine");
  }
  auto kernel = a.k <= 2 ? moek::combine_kernel<2, 4> : a.k <= 4 ? moek::combine_kernel<4, 2> : moek::combine_kernel<8, 2>;
  return launched(launch(kernel, a, 2 * kMoeSegments, moek::kCombineThreads, 0, stream, a), "moe combine");
}

Status launch_moe_combine_grad(const void* g_out, const void* y, const float* w, const int* send_pos, void* g_y, float* g_w, int rows, int T, int k,
                               int d, cudaStream_t stream) {
  if (T == 0) return kSuccess;
  return launched(launch_overlapped(moek::combine_grad_kernel, dim3(T), dim3(moek::kGradThreads), 0, stream, (const char*)g_out, (const char*)y, w, send_pos,
                                    (char*)g_y, g_w, rows, T, k, d), "moe combine gradient");
}

Status launch_moe_input_grad(const void* g_rows, const int* send_pos, const int* idx, const void* g_logits, const void* router, void* g_x, int rows, int T,
                             int k, int d, int E, cudaStream_t stream) {
  return launched(launch_overlapped(moek::input_grad_kernel, dim3(2 * kMoeSegments), dim3(moek::kCombineThreads), 0, stream, (const char*)g_rows, send_pos, idx,
                                    (const __nv_bfloat16*)g_logits, (const char*)router, (char*)g_x, rows, T, k, d, E), "moe input gradient");
}

template <typename K>
static Status coop(K kernel, dim3 grid, int threads, size_t smem, void** params, cudaStream_t stream, const char* what) {
  return launched(cudaLaunchCooperativeKernel((const void*)kernel, grid, dim3(threads), params, smem, stream), what);
}

Status launch_moe_dispatch_emu(const MoeArgs* host_all, const MoeArgs* dev_all, int nranks, cudaStream_t stream) {
  const int segs = 8;
  moek::count_kernel_emu<<<dim3(segs, nranks), moek::kThreads, 0, stream>>>(dev_all);
  AMEM_TRY(launched(cudaGetLastError(), "moe count(emu)"));
  int segments = segs;
  void* p2[] = {(void*)&dev_all, (void*)&segments};
  AMEM_TRY(coop(moek::plan_kernel_emu, dim3(1, nranks), moek::kThreads, 0, p2, stream, "moe plan(emu)"));
  void* p3[] = {(void*)&dev_all};
  return coop(moek::scatter_kernel_emu, dim3(segs, nranks), moek::kThreads, moek::whist_bytes(host_all[0].E), p3, stream, "moe scatter(emu)");
}

Status launch_moe_combine_emu(const MoeArgs*, const MoeArgs* dev_all, int nranks, cudaStream_t stream) {
  void* p[] = {(void*)&dev_all};
  return coop(moek::combine_kernel_emu, dim3(8, nranks), moek::kCombineThreads, 0, p, stream, "moe combine(emu)");
}

}  // namespace amem
