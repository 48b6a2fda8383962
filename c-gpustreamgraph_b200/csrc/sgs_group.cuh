// sgs_group.cuh -- query groups: up to GMAX integer queries (BFS / SSSP / CC,
// any sources) relaxed together over one edge stream.
//
// Layout: st[v * S + lane] u64 packed (value << 32 | parent), S = 1, 2 or 4,
// so one vertex's states share one 32-B sector and a random access to a
// destination serves every lane.  Lane masks mask[k][v] (u32, three rotating
// buffers) record which lanes improved v in a round; the thread whose
// atomicOr turns the mask non-zero appends v, which replaces per-query
// de-duplication stamps.  Round r reads mask[r%3], writes mask[(r+1)%3] and
// clears the masks of frontier r-1 in mask[(r+2)%3], which round r+1 writes
// next; frontier buffers rotate the same way, so no grid barrier is needed.
//
// Reference semantics per lane are those of the single-query ops
// (hybrid_sssp.cu:97-118 min relaxation, hybrid_cc.cu:96-110 label
// propagation, reset_del_edges / SyncPushDDB_del parent-tree invalidation,
// driver.cuh:398-430 and :1985-2031).
#pragma once
#include <cooperative_groups.h>

#include <algorithm>

#include "sgs_device.cuh"
#include "sgs_segmap.cuh"

namespace sgs {

constexpr int GMAX = 4;
constexpr int GCHUNK = 512;  // entries staged per chunk by group_map

struct LaneAlgo {
  uint32_t packed;  // 8 bits per lane: A_BFS / A_SSSP / A_CC
  // the same as lane bit masks (bit q = lane q), so a relaxation picks a
  // lane's step from kernel-parameter constants instead of decoding `packed`:
  // candidate = source value + (w: the edge weight, inc: 1, cc: 0)
  uint32_t cc, w, inc;
  __device__ __forceinline__ int at(int q) const { return (packed >> (8 * q)) & 0xFF; }
  static LaneAlgo of(uint32_t packed) {
    LaneAlgo a{packed, 0, 0, 0};
    for (int q = 0; q < 4; ++q) {
      const uint32_t k = (packed >> (8 * q)) & 0xFF;
      if (k == A_CC) a.cc |= 1u << q;
      else if (k == A_SSSP) a.w |= 1u << q;
      else a.inc |= 1u << q;
    }
    return a;
  }
};

template <int S>
struct GPay {
  uint64_t off;
  uint32_t mask;
  uint32_t val[S];
};

// S u32 values of vertex v (one 16-B load for S = 4).
template <int S>
__device__ __forceinline__ void load_vals(const uint32_t *val, uint32_t v, uint32_t (&o)[S]) {
  if constexpr (S == 4) {
    const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(val + (uint64_t)v * 4));
    o[0] = x.x; o[1] = x.y; o[2] = x.z; o[3] = x.w;
  } else if constexpr (S == 2) {
    const uint2 x = __ldcg(reinterpret_cast<const uint2 *>(val + (uint64_t)v * 2));
    o[0] = x.x; o[1] = x.y;
  } else {
    o[0] = __ldcg(val + v);
  }
}

// How a narrow group's repair starts, decided on the device from the reset
// counts of the invalidation (per lane), the same in every kernel involved:
//  NONE        nothing was reset: only the inserted edges are relaxed;
//  RESTRICTED  round 0 walks every reached vertex's edges but relaxes only
//              those into reset vertices (k_group_sweep), and the inserted
//              edges are relaxed beside it: all other edges already satisfy
//              value(u) + w >= value(v), so these hold every violated one;
//  FULL        round 0 relaxes every edge (group_map), when more than
//              `restrict_max` (lane, vertex) pairs were reset -- the filter
//              then passes so many edges that testing them costs more.
enum RepairMode : int { REPAIR_NONE = 0, REPAIR_RESTRICTED = 1, REPAIR_FULL = 2 };
__device__ __forceinline__ int repair_mode(const unsigned long long *resets, uint32_t lanes,
                                           unsigned long long restrict_max) {
  unsigned long long n = 0;
#pragma unroll
  for (int q = 0; q < GMAX; ++q)
    if (lanes >> q & 1u) n += __ldg(resets + q);
  return n == 0 ? REPAIR_NONE : n <= restrict_max ? REPAIR_RESTRICTED : REPAIR_FULL;
}

// Clears the masks of the previous frontier (grid-stride, all threads).
__device__ __forceinline__ void clear_prev_masks(const uint32_t *vtx, const unsigned long long *cnt,
                                                 uint32_t *mask) {
  if (!cnt) return;
  const uint32_t n = (uint32_t)(__ldcg(cnt) >> CNT_SHIFT);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    mask[__ldcg(&vtx[i])] = 0;
}

// Relaxation of every active lane of every source over its out-edges.  The
// u32 mirror `val` filters candidates with one 16-B read per destination; a
// candidate below it lowers the mirror first and, if that strictly lowered
// it, the packed (value,parent) word (relax_mirror_packed: equal candidates
// never swap a parent).
//
// Per entry the payload holds each lane's candidate base -- the source's
// value, plus 1 in BFS lanes -- and INF32 in the lanes that do not push, so
// the per-edge test is compare-only: candidate = base (+ the weight in SSSP
// lanes, saturating at INF32) against the destination's mirror.  Most edges
// of a sweep improve nothing; only the quads with some candidate below the
// mirror take the atomic path.
template <int S>
struct RPay {
  uint64_t off;
  uint32_t mask;     // lanes that push from this vertex
  uint32_t base[S];  // candidate base per lane (INF32: the lane does not push)
};

template <int S>
struct GroupRelaxOp {
  static constexpr int kBlocks = 4;
  static constexpr bool kResets = false;
  using Payload = RPay<S>;
  GraphView g;
  unsigned long long *st;
  uint32_t *val;
  const uint32_t *m_in;
  uint32_t *m_out;
  LaneAlgo algo;
  uint32_t any_w;  // some lane reads stored weights
  __device__ __forceinline__ Payload load(uint32_t v) const {
    Payload p;
    p.off = g.off[v];
    p.mask = __ldcg(&m_in[v]);
    uint32_t x[S];
    load_vals<S>(val, v, x);
    // a BFS/SSSP lane that has not reached v pushes nothing: drop it here,
    // once per entry, instead of testing it for every edge.  A reached BFS
    // value is below INF32, so value + 1 does not wrap.
#pragma unroll
    for (int q = 0; q < S; ++q) {
      const bool on = (p.mask >> q & 1u) && (x[q] != INF32 || (algo.cc >> q & 1u));
      if (!on) p.mask &= ~(1u << q);
      p.base[q] = on ? x[q] + (algo.inc >> q & 1u) : INF32;
    }
    return p;
  }
  // The quad's ids (and weights), loaded one step ahead by group_map.
  struct Quad {
    uint4 ids, ws;
  };
  // H: the graph has a host tier (blocks may be host-resident or cached)
  template <bool H>
  __device__ __forceinline__ Quad fetch(const Payload &p, uint32_t j0) const {
    Quad q;
    if constexpr (H) {
      q.ids = ld_quad_stream(adj_at(g, p.off, j0));
      q.ws = any_w ? ld_quad_stream(wgt_at(g, p.off, j0)) : make_uint4(1, 1, 1, 1);
    } else {
      q.ids = ld_quad_stream(g.adj_d + p.off + j0);
      q.ws = any_w ? ld_quad_stream(g.wgt_d + p.off + j0) : make_uint4(1, 1, 1, 1);
    }
    return q;
  }
  // candidate of lane q for an edge of weight w: base + w in SSSP lanes,
  // saturating (min(base, INF32 - w) + w), else base; INF32 is never below
  // a mirror value
  __device__ __forceinline__ uint32_t cand_of(uint32_t base, uint32_t w, int q) const {
    const uint32_t wq = w & (0u - (algo.w >> q & 1u));
    return min(base, ~wq) + wq;
  }
  __device__ __forceinline__ uint32_t weight_of(const uint4 &ws, int k, uint32_t u, uint32_t d) const {
    return g.wmode == W_EXPLICIT ? quad_at(ws, k) : g.wmode == W_SYNTH ? (u + d) % 128u + 1u : 1u;
  }
  // Returns a 4-bit mask of destinations to append; dst[] holds them, sl[] their
  // slots.
  __device__ __forceinline__ uint32_t visit4(uint32_t u, const Payload &pr, uint32_t j0, uint32_t len,
                                             const Quad &qd, uint32_t (&dst)[4], uint32_t (&sl)[4],
                                             uint32_t *) const {
    const uint4 ids = qd.ids;
    const uint4 ws = qd.ws;
    uint32_t okm = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      dst[k] = quad_at(ids, k);
      if (j0 + k < len && dst[k] != SGS_TOMB) okm |= 1u << k;
    }
    uint32_t cur[4][S];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (okm >> k & 1u) load_vals<S>(val, dst[k], cur[k]);
    // compare-only pass: bit 4k+q = lane q's candidate is below the mirror
    // of destination k
    uint32_t lt = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (!(okm >> k & 1u)) continue;
      const uint32_t w = weight_of(ws, k, u, dst[k]);
#pragma unroll
      for (int q = 0; q < S; ++q)
        lt |= (cand_of(pr.base[q], w, q) < cur[k][q] ? 1u : 0u) << (4 * k + q);
    }
    if (!lt) return 0;
    // The atomics go out together, then their answers are looked at: with a
    // wait after each (up to 16 per quad, one lane's improvement holding up the
    // whole warp) a round's length was that chain.  (With units of 1024 slots
    // and one append per CTA at a round's end, scale 16, 20,000 updates:
    // relaxation rounds 140 -> 91 us, invalidation rounds 148 -> 93 us.)
    uint32_t old[4][S];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t w = weight_of(ws, k, u, dst[k]);
#pragma unroll
      for (int q = 0; q < S; ++q) {
        old[k][q] = 0;
        if (lt >> (4 * k + q) & 1u)
          old[k][q] = atomicMin(&val[(uint64_t)dst[k] * S + q], cand_of(pr.base[q], w, q));
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) sl[k] = lt >> (4 * k) & 0xFu ? g.slots[dst[k]] : 0u;
    uint32_t app = 0, seen[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t w = weight_of(ws, k, u, dst[k]);
      uint32_t bits = 0;
#pragma unroll
      for (int q = 0; q < S; ++q) {
        const uint32_t cand = cand_of(pr.base[q], w, q);
        if (old[k][q] > cand) {  // strictly lowered (0 where no candidate was offered)
          atomicMin(&st[(uint64_t)dst[k] * S + q], ((unsigned long long)cand << 32) | u);
          bits |= 1u << q;
        }
      }
      seen[k] = 1u;
      if (bits && sl[k]) seen[k] = atomicOr(&m_out[dst[k]], bits);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) app |= (seen[k] == 0u ? 1u : 0u) << k;
    return app;
  }
};

// S packed words of vertex v (two 16-B loads for S = 4).
template <int S>
__device__ __forceinline__ void load_row(const unsigned long long *st, uint32_t v, unsigned long long (&o)[S]) {
  if constexpr (S == 4) {
    const ulonglong2 a = __ldcg(reinterpret_cast<const ulonglong2 *>(st + (uint64_t)v * 4));
    const ulonglong2 b = __ldcg(reinterpret_cast<const ulonglong2 *>(st + (uint64_t)v * 4 + 2));
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
  } else {
#pragma unroll
    for (int q = 0; q < S; ++q) o[q] = __ldcg(st + (uint64_t)v * S + q);
  }
}

// Parent-tree invalidation per lane: a child whose lane-q parent is u (and u
// was reset in lane q) is reset exactly once (CAS on the packed word); the
// mirror is reset with it.
template <int S>
struct GroupInvalidateOp {
  static constexpr int kBlocks = 3;
  static constexpr bool kResets = true;
  struct Payload {
    uint64_t off;
    uint32_t mask;
    uint32_t pad;
  };
  GraphView g;
  unsigned long long *st;
  uint32_t *val;
  const uint32_t *m_in;
  uint32_t *m_out;
  LaneAlgo algo;
  unsigned long long *inval;  // [GMAX] per-lane reset counts
  uint32_t *mark;             // bitmap of reset vertices (may be null)
  __device__ __forceinline__ Payload load(uint32_t v) const {
    Payload p;
    p.off = g.off[v];
    p.mask = __ldcg(&m_in[v]);
    p.pad = 0;
    return p;
  }
  struct Quad {
    uint4 ids;
  };
  template <bool H>
  __device__ __forceinline__ Quad fetch(const Payload &p, uint32_t j0) const {
    if constexpr (H) return Quad{ld_quad_stream(adj_at(g, p.off, j0))};
    else return Quad{ld_quad_stream(g.adj_d + p.off + j0)};
  }
  __device__ __forceinline__ uint32_t visit4(uint32_t u, const Payload &p, uint32_t j0, uint32_t len,
                                             const Quad &qd, uint32_t (&dst)[4], uint32_t (&sl)[4],
                                             uint32_t *resets) const {
    const uint4 ids = qd.ids;
    uint32_t okm = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      dst[k] = quad_at(ids, k);
      if (j0 + k < len && dst[k] != SGS_TOMB) okm |= 1u << k;
    }
    // rows, then the resets, then the masks: each kind together (see GroupRelaxOp)
    unsigned long long row[4][S];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (okm >> k & 1u) load_row<S>(st, dst[k], row[k]);
    uint32_t hit = 0;  // bit 4k+q: lane q's parent of destination k is u
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int q = 0; q < S; ++q)
        if ((okm >> k & 1u) && (p.mask >> q & 1u) && (uint32_t)row[k][q] == u) hit |= 1u << (4 * k + q);
    if (!hit) return 0;
    unsigned long long was[4][S];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int q = 0; q < S; ++q) {
        was[k][q] = 0;
        if (hit >> (4 * k + q) & 1u)
          was[k][q] = atomicCAS(&st[(uint64_t)dst[k] * S + q], row[k][q],
                                algo.at(q) == A_CC ? (((unsigned long long)dst[k] << 32) | INF32) : ~0ull);
      }
    uint32_t seen[4], app = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) sl[k] = hit >> (4 * k) & 0xFu ? g.slots[dst[k]] : 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t bits = 0;
#pragma unroll
      for (int q = 0; q < S; ++q) {
        if (!(hit >> (4 * k + q) & 1u) || was[k][q] != row[k][q]) continue;
        val[(uint64_t)dst[k] * S + q] = algo.at(q) == A_CC ? dst[k] : INF32;
        bits |= 1u << q;
        atomicAdd(&resets[q], 1u);
      }
      if (bits && mark) bit_set(mark, dst[k]);
      seen[k] = 1u;
      if (bits && sl[k]) seen[k] = atomicOr(&m_out[dst[k]], bits);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) app |= (seen[k] == 0u ? 1u : 0u) << k;
    return app;
  }
};

// Load-balanced map for group ops (same unit/chunk scheme as seg_map).
// Edges are attributed per entry: the CTA whose range holds an entry's first
// position adds live[v] for every lane of its mask, which counts exactly the
// (query, edge) pairs relaxed.  The kernel also clears the previous
// frontier's masks.
// (Op::kBlocks: resident CTAs per SM that the registers are budgeted for; 4 of
// 64 registers for the relaxation, 3 for the invalidation, which holds four
// 32-B rows per thread.)
// H = false when every block is in HBM (no host tier): the host-tier logic
// (hotness, cache lookups, link accounting) is compiled out.
template <class Op, bool H>
__device__ __forceinline__ void group_map_body(FrontierView in, FrontierView out, const Op &op,
                                               const uint32_t *prev_vtx,
                                               const unsigned long long *prev_cnt, uint32_t *prev_mask,
                                               unsigned long long *lane_edges,
                                               unsigned long long *edge_stat,
                                               unsigned long long *host_stat, uint64_t packed) {
  using P = typename Op::Payload;
  constexpr int GC = GCHUNK;
  __shared__ uint64_t s_eb[GC + 1];
  __shared__ uint32_t s_len[GC];
  __shared__ P s_pay[GC];
  __shared__ uint32_t s_vtx[GC];
  __shared__ unsigned long long s_lane[GMAX];
  __shared__ unsigned long long s_host, s_all;  // host-tier slots read over the link / owned
  __shared__ uint32_t s_reset[GMAX];            // resets of an invalidation, per lane
  __shared__ uint2 s_queue[RELAX_THREADS / 32][WarpQueue::CAP];
  WarpQueue queue(s_queue[threadIdx.x >> 5]);
  if (threadIdx.x < GMAX) {
    s_lane[threadIdx.x] = 0;
    s_reset[threadIdx.x] = 0;
  }
  if (threadIdx.x == 0) s_host = s_all = 0;
  uint32_t host_acc = 0;
  const uint32_t n = (uint32_t)(packed >> CNT_SHIFT);
  const uint64_t T = packed & EDGE_MASK;
  const uint64_t nunits = (T + UNIT - 1) / UNIT;
  const uint64_t ub = (uint64_t)blockIdx.x * nunits / gridDim.x;
  const uint64_t ue = (uint64_t)(blockIdx.x + 1) * nunits / gridDim.x;
  if (n != 0 && ub < ue) {
    const uint64_t E0 = ub * UNIT;
    const uint64_t E1 = min(ue * (uint64_t)UNIT, T);
    uint32_t s = __ldcg(&in.ustart[ub]);
    for (;;) {
      __syncthreads();
      bool host = false;  // this thread staged a host-tier entry
      uint32_t lane_acc[GMAX] = {0, 0, 0, 0};  // (query, edge) pairs of owned entries
#pragma unroll
      for (int h = 0; h < GC / RELAX_THREADS; ++h) {
        const uint32_t t = threadIdx.x + h * RELAX_THREADS;
        const uint32_t idx = s + t;
        const uint64_t eb = idx < n ? __ldcg((const unsigned long long *)&in.ebase[idx]) : T;
        s_eb[t] = eb;
        if (t == 0) {
          const uint32_t j = s + GC;
          s_eb[GC] = j < n ? __ldcg((const unsigned long long *)&in.ebase[j]) : T;
        }
        if (idx < n && eb < E1) {
          const uint32_t v = __ldcg(&in.vtx[idx]);
          s_vtx[t] = v;
          s_len[t] = __ldcg(&in.len[idx]);
          P pay = op.load(v);
          if constexpr (H) {
            if (pay.off & HOST_BIT) {
              host = true;
              if (eb >= E0) {
                hot_bump(op.g, v, pay.off);
                if (op.g.cstat) atomicAdd(&s_all, (unsigned long long)s_len[t]);
              }
              pay.off = resolve_block(op.g, pay.off, s_len[t]);
            }
          }
          s_pay[t] = pay;
          if (eb >= E0 && pay.mask) {
            const uint32_t l = op.g.live[v];
#pragma unroll
            for (int q = 0; q < GMAX; ++q) lane_acc[q] += (pay.mask >> q & 1u) ? l : 0u;
          }
        }
      }
      // the chunk's pair counts go to shared memory now, so no register
      // holds them through the walk
#pragma unroll
      for (int q = 0; q < GMAX; ++q) {
        const uint32_t x = warp_sum(lane_acc[q]);
        if ((threadIdx.x & 31) == 0 && x) atomicAdd(&s_lane[q], (unsigned long long)x);
      }
      // the barrier also tells every thread whether the chunk holds
      // host-tier entries (only then does the walk account host reads)
      bool chunk_host = false;
      if constexpr (H) chunk_host = __syncthreads_or(host) != 0;
      else __syncthreads();
      const uint64_t lo = max(E0, s_eb[0]);
      const uint64_t hi = min(E1, s_eb[GC]);
      // Each warp walks its own contiguous share of the chunk's positions,
      // one window of 32 quads (128 slots) per step, lane i on quad i of the
      // window (coalesced 512-B id reads).  Owners need no search: lane j
      // holds the start of entry s0 + j (s0 = owner of the window's first
      // quad), every start inside the window sets bit (start - window) / 4
      // of a warp-wide OR, and a lane's owner is s0 plus the set bits at or
      // below its quad.  This relies on every frontier entry having at least
      // one slot (every append site checks it), so a window meets at most 32
      // entries and no two starts share a bit.  The same bits give the next
      // window's first owner.  Software pipeline: the next window's owners
      // and id loads are issued before the current window's state reads.
      constexpr uint32_t NW = RELAX_THREADS / 32;
      const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
      const uint64_t nq = hi > lo ? (hi - lo) >> 2 : 0;
      uint64_t wq = (lo >> 2) + nq * wid / NW;  // this warp's share [wq, wqe) in quads
      const uint64_t wqe = (lo >> 2) + nq * (wid + 1) / NW;
      if (wq < wqe) {
        int s0;
        {  // owner of the share's first quad: one warp-uniform search per chunk
          const uint64_t e = wq << 2;
          int a = 0, b = GC - 1;
          while (a < b) {
            const int m = (a + b + 1) >> 1;
            if (s_eb[m] <= e) a = m;
            else b = m - 1;
          }
          s0 = a;
        }
        // Owner and first slot of this lane's quad in the window at quad q
        // (called for consecutive windows, all lanes together); true when
        // the quad holds slots.  Leaves s0 at the next window's first owner.
        auto window = [&](uint64_t q, int &own, uint32_t &j0) -> bool {
          const uint64_t p0 = q << 2, pe = p0 + 4 * 32;
          const int j = s0 + (int)lane;
          const uint64_t bj = j <= GC ? s_eb[j] : ~0ull;
          const uint32_t bit = (lane >= 1 && bj < pe) ? 1u << (uint32_t)((bj - p0) >> 2) : 0u;
          const uint32_t m = __reduce_or_sync(0xFFFFFFFFu, bit);
          own = s0 + __popc(m & (0xFFFFFFFFu >> (31 - lane)));
          int ns = s0 + __popc(m);
          if (ns < GC && s_eb[ns + 1] <= pe) ++ns;  // an entry starting exactly at pe
          s0 = ns;
          j0 = (uint32_t)(p0 + 4 * lane - s_eb[own]);
          return q + lane < wqe && j0 < s_len[own];
        };
        int oc = 0;
        uint32_t jc = 0;
        typename Op::Quad qc{};
        bool hc = window(wq, oc, jc);
        if (hc) qc = op.template fetch<H>(s_pay[oc], jc);
        for (; wq < wqe; wq += 32) {
          int on = 0;
          uint32_t jn = 0;
          typename Op::Quad qn{};
          bool hn = false;
          if (wq + 32 < wqe) {
            hn = window(wq + 32, on, jn);
            if (hn) qn = op.template fetch<H>(s_pay[on], jn);
          }
          uint32_t app = 0;
          uint32_t dst[4] = {0, 0, 0, 0}, sl[4] = {0, 0, 0, 0};
          if (hc) {
            app = op.visit4(s_vtx[oc], s_pay[oc], jc, s_len[oc], qc, dst, sl, s_reset);
            if (H && chunk_host) {
              const uint64_t o = s_pay[oc].off;
              if ((o & HOST_BIT) && cache_line(op.g, (o & OFF_MASK) + jc) == NO_LINE)
                host_acc += min(4u, s_len[oc] - jc);
            }
          }
          oc = on;
          jc = jn;
          qc = qn;
          hc = hn;
          queue.push4(out, app, dst, sl);
        }
      }
      if (s_eb[GC] >= E1 || s + GC >= n) break;
      s += GC;
    }
    queue.template finish<RELAX_THREADS>(out);
  }
  // (after the walk: its loads would delay a CTA that has edges, and most have
  // none in the small rounds)
  clear_prev_masks(prev_vtx, prev_cnt, prev_mask);
  const unsigned long long hs = warp_sum((unsigned long long)host_acc);
  if ((threadIdx.x & 31) == 0 && hs) atomicAdd(&s_host, hs);
  __syncthreads();
  if (threadIdx.x < GMAX && s_lane[threadIdx.x]) {
    if (lane_edges) atomicAdd(&lane_edges[threadIdx.x], s_lane[threadIdx.x]);
  }
  // (one global atomic per CTA and lane; one per reset, all on the group's few
  // counters, was most of a large snapshot's first rounds)
  if constexpr (Op::kResets)
    if (threadIdx.x < GMAX && s_reset[threadIdx.x])
      atomicAdd(&op.inval[threadIdx.x], (unsigned long long)s_reset[threadIdx.x]);
  if (threadIdx.x == 0 && edge_stat) {
    unsigned long long all = 0;
#pragma unroll
    for (int q = 0; q < GMAX; ++q) all += s_lane[q];
    if (all) atomicAdd(edge_stat, all);
  }
  if (threadIdx.x == 0 && s_host && host_stat) atomicAdd(host_stat, s_host);
  if (threadIdx.x == 0 && op.g.cstat) {
    if (s_all) atomicAdd(&op.g.cstat[0], s_all);
    if (s_host) atomicAdd(&op.g.cstat[1], s_host);
  }
  __syncthreads();  // shared state is reused when the body runs again
}

template <class Op, bool H>
__global__ void __launch_bounds__(RELAX_THREADS, Op::kBlocks)
    group_map(FrontierView in, FrontierView out, Op op, const uint32_t *prev_vtx,
              const unsigned long long *prev_cnt, uint32_t *prev_mask,
              unsigned long long *lane_edges, unsigned long long *edge_stat,
              unsigned long long *host_stat, uint32_t lanes = 0,
              const unsigned long long *resets = nullptr, unsigned long long restrict_max = 0) {
  // round 0 of a repair that k_group_sweep has done
  if (resets && repair_mode(resets, lanes, restrict_max) == REPAIR_RESTRICTED) return;
  group_map_body<Op, H>(in, out, op, prev_vtx, prev_cnt, prev_mask, lane_edges, edge_stat, host_stat,
                        __ldcg((const unsigned long long *)in.counter));
}

// The three rotating frontier buffers, their counters and lane masks, as one
// persistent launch sees them: round r reads buffer r % 3 / cnt[r] and masks
// r % 3, and writes buffer (r+1) % 3 / cnt[r+1].
template <class M>
struct RoundBufs {
  uint32_t *vtx[3];
  uint32_t *len[3];
  uint64_t *ebase[3];
  uint32_t *ustart[3];
  unsigned long long *cnt;
  M *mask[3];
  uint32_t ucap;
  __device__ __forceinline__ FrontierView view(uint32_t r) const {
    FrontierView f;
    f.vtx = vtx[r % 3];
    f.len = len[r % 3];
    f.ebase = ebase[r % 3];
    f.ustart = ustart[r % 3];
    f.counter = (uint64_t *)(cnt + r);
    f.ucap = ucap;
    return f;
  }
};

// Rounds r0, r0+1, ... of a phase in one cooperative launch: round r, a
// grid-wide barrier (cooperative_groups grid sync; the cooperative launch
// makes every block resident), then the next round unless round r appended
// nothing.  The masks of the last non-empty frontier are cleared before the
// kernel returns; *rounds_out = the first empty frontier's index (or
// max_rounds when the limit is hit).
template <class Op, bool H>
__global__ void __launch_bounds__(RELAX_THREADS, Op::kBlocks)
    group_rounds(RoundBufs<uint32_t> rb, Op op, uint32_t r0, uint32_t max_rounds,
                 unsigned long long *lane_edges, unsigned long long *rstat, unsigned long long *hstat,
                 uint32_t *rounds_out) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  uint32_t r = r0;
  bool conv = false;
  uint64_t packed = __ldcg(rb.cnt + r0);
  for (; r < max_rounds; ++r) {
    Op o = op;
    o.m_in = rb.mask[r % 3];
    o.m_out = rb.mask[(r + 1) % 3];
    const bool hp = r >= 1;
    group_map_body<Op, H>(rb.view(r), rb.view(r + 1), o, hp ? rb.vtx[(r - 1) % 3] : nullptr,
                   hp ? rb.cnt + r - 1 : nullptr, hp ? rb.mask[(r - 1) % 3] : nullptr, lane_edges,
                   rstat + r, hstat + r, packed);
    grid.sync();
    packed = __ldcg(rb.cnt + r + 1);
    if ((packed >> CNT_SHIFT) == 0) {
      conv = true;
      ++r;
      break;
    }
  }
  // r: the first empty frontier (converged) or max_rounds
  if (r >= 1) clear_prev_masks(rb.vtx[(r - 1) % 3], rb.cnt + r - 1, rb.mask[(r - 1) % 3]);
  if (!conv) clear_prev_masks(rb.vtx[r % 3], rb.cnt + r, rb.mask[r % 3]);
  if (blockIdx.x == 0 && threadIdx.x == 0) *rounds_out = r;
}

// ---------------------------------------------------------------------------
// Group frontier builders
// ---------------------------------------------------------------------------
template <int S>
__global__ void k_group_init_lane(unsigned long long *st, uint32_t *val, uint32_t nv, int lane,
                                  int algo, uint32_t source) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride) {
    unsigned long long s;
    if (algo == A_CC) s = (v << 32) | INF32;
    else s = v == source ? (unsigned long long)INF32 : ~0ull;
    st[v * S + lane] = s;
    val[v * S + lane] = (uint32_t)(s >> 32);
  }
}

// Every vertex with a non-empty block; mask = selected lanes whose value is
// finite there (CC lanes always).  One writer per vertex: plain stores.
// With `resets`, only in repair mode FULL.
template <int S>
__global__ void k_group_dense(GraphView g, const uint32_t *val, uint32_t lanes,
                              LaneAlgo algo, uint32_t *m_out, FrontierView out,
                              const unsigned long long *resets = nullptr,
                              unsigned long long restrict_max = 0) {
  if (resets && repair_mode(resets, lanes, restrict_max) != REPAIR_FULL) return;
  // eight consecutive vertices per thread, one block append per 2048
  constexpr int N = 8;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * N;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x * N; b < g.nv; b += stride) {
    const uint64_t v0 = b + (uint64_t)threadIdx.x * N;
    bool want[N];
    uint32_t d[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint64_t v = v0 + i;
      want[i] = false;
      d[i] = 0;
      if (v < g.nv) {
        d[i] = g.slots[v];
        if (d[i]) {
          uint32_t blk[S];
          load_vals<S>(val, (uint32_t)v, blk);
          uint32_t m = 0;
#pragma unroll
          for (int q = 0; q < S; ++q)
            if ((lanes >> q & 1u) && (algo.at(q) == A_CC || blk[q] != INF32)) m |= 1u << q;
          if (m) {
            m_out[v] = m;
            want[i] = true;
          }
        }
      }
    }
    frontier_append_block_n<N>(out, want, (uint32_t)v0, d);
  }
}

// Coarse form of the reset bitmap for k_group_sweep's shared-memory filter: bit
// b = some vertex of [b << shift, (b + 1) << shift) was reset.
__global__ void k_fold_bits(const uint32_t *bits, uint32_t nwords, uint32_t shift, uint32_t *coarse,
                            uint32_t cwords) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < cwords; c += gridDim.x * blockDim.x) {
    uint32_t o = 0;
    for (uint32_t b = 0; b < 32; ++b) {
      const uint64_t v0 = ((uint64_t)c * 32 + b) << shift;
      uint32_t any = 0;
      if (shift >= 5) {
        for (uint64_t w = v0 >> 5; w < (v0 >> 5) + (1u << (shift - 5)) && w < nwords; ++w) any |= bits[w];
      } else if ((v0 >> 5) < nwords) {
        any = bits[v0 >> 5] >> (v0 & 31) & ((1u << (1u << shift)) - 1u);
      }
      if (any) o |= 1u << b;
    }
    coarse[c] = o;
  }
}

// Round 0 of a narrow group's repair in mode RESTRICTED: a walk of the ids of
// every reached vertex's block in which only the edges into reset vertices are
// relaxed.
//
// The full sweep reads a random 16-B mirror row per slot, and that gather, not
// the id stream, sets its time.  Here a slot costs one bit of a filter in
// shared memory: the reset bitmap, for up to 2^20 vertices exactly, above that
// one bit per 2^shift consecutive vertices, with the exact bitmap probed for
// the slots that pass.  What passes goes through per-warp queues and is
// handled 32 edges at a time, so the few edges per window that need the rows
// of both ends do not stall the walk with mostly idle warps.  The walk is then
// bound by the instructions per slot, so it goes over the vertices themselves,
// 32 consecutive ones per warp and step, instead of a frontier built and read
// back (that was 0.2 ms of scale 24's 1.9): their blocks' starts come from
// a warp scan, a quad's owner from the OR of starts (as in group_map, in 32
// bits).  Blocks of more than SWEEP_BIG slots are cut into slices, listed by the
// first phase and walked by all warps after a grid barrier, without owners.
// Warps take vertices from a counter, since blocks differ widely in size.
// One CTA of 32 warps per SM (the filter takes 128 KB).
// Scale 24, three lanes, a million updates: 1.06 ms; 1.55 and 0.26 for the
// frontier when it took its blocks from one, 1.67 and 0.21 as the full sweep.
// Scale 16: 38 us against 37 + 12.  With the blocks behind the host link
// (2^20 vertices, 0.35 of the graph in HBM) 1.36 ms either way: the link.
constexpr int SWEEP_THREADS = 1024;
constexpr uint32_t SWEEP_FILTER_BITS = 1u << 20;
constexpr uint32_t SWEEP_SLICE = 1024;
constexpr uint32_t SWEEP_BIG = 256;  // a step's 32 blocks then hold 64 windows at most
struct SweepWarp {
  uint64_t off[32];
  uint32_t eb[33], len[32], vtx[32];
  // queue 1: slots that passed the filter; queue 2: edges into reset vertices
  // (up to 31 waiting, 32 new)
  uint32_t d1[63], s1[63], j1[63];
  uint32_t d2[63], s2[63], j2[63];
  uint2 app[WarpQueue::CAP1];
};
inline size_t sweep_smem(uint32_t filter_words) {  // (a power of two, at least 16)
  return sizeof(SweepWarp) * (SWEEP_THREADS / 32) + (size_t)filter_words * 4;
}
// Counters (zero before the launch) and lists of a sweep.
struct SweepCtx {
  const uint32_t *bits, *coarse;  // reset bitmap and its folded form (shift > 0)
  uint32_t filter_words, filter_mask, shift, lanes;  // words given; words kept - 1 (all ones)
  const unsigned long long *resets;
  unsigned long long restrict_max;
  unsigned long long *next;       // next vertex to take
  unsigned long long *n_slices;   // slices listed
  unsigned long long *walked;     // packed (vertices << CNT_SHIFT | padded slots)
  uint2 *slices;                  // (vertex, slice)
  uint32_t batch, step;           // vertices taken at a time, and walked at a time (at most 32)
  unsigned long long *lane_edges, *edge_stat, *host_stat;
};

template <bool H>
__global__ void __launch_bounds__(SWEEP_THREADS, 1)
    k_group_sweep(FrontierView out, GroupRelaxOp<GMAX> op, SweepCtx c) {
  if (repair_mode(c.resets, c.lanes, c.restrict_max) != REPAIR_RESTRICTED) return;
  extern __shared__ __align__(16) unsigned char s_raw[];
  SweepWarp &sw = reinterpret_cast<SweepWarp *>(s_raw)[threadIdx.x >> 5];
  uint32_t *filter = reinterpret_cast<uint32_t *>(s_raw + sizeof(SweepWarp) * (SWEEP_THREADS / 32));
  // (its length is a power of two, so that any id, a tombstone too, can be
  // masked into it; what a false hit of that kind leads to checks the id)
  {
    const uint32_t *f_src = c.shift ? c.coarse : c.bits;
    for (uint32_t i = threadIdx.x; i <= c.filter_mask; i += SWEEP_THREADS)
      filter[i] = i < c.filter_words ? f_src[i] : 0u;
  }
  __syncthreads();
  const GraphView &g = op.g;
  const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u, full = 0xFFFFFFFFu;
  const uint32_t shift = c.shift, shift5 = shift + 5, mask = c.filter_mask;
  WarpQueue queue(sw.app);
  uint32_t evald = 0, host_acc = 0, n1 = 0, n2 = 0;  // n1, n2: queued (warp-uniform)
  unsigned long long host_all = 0, walked = 0, edges[GMAX] = {};
  // Takes the last 32 (or fewer) of queue 1: relaxes them when the filter is
  // exact, else probes the bitmap, queues those that lead into reset vertices and
  // relaxes these 32 at a time.  `all`: both queues, to the end.
  auto drain = [&](bool all) {
    const uint32_t *qd = shift ? sw.d2 : sw.d1, *qs = shift ? sw.s2 : sw.s1, *qj = shift ? sw.j2 : sw.j1;
#pragma unroll 1
    do {
      uint32_t d = 0, u = 0, j = 0;
      if (shift && n1) {
        const uint32_t k = min(n1, 32u);
        bool on = false;
        if (lane < k) {
          d = sw.d1[n1 - k + lane];
          u = sw.s1[n1 - k + lane];
          j = sw.j1[n1 - k + lane];
          on = d != SGS_TOMB && (__ldg(c.bits + (d >> 5)) >> (d & 31) & 1u);
        }
        n1 -= k;
        const uint32_t m = __ballot_sync(full, on);
        if (on) {
          const uint32_t at = n2 + __popc(m & below);
          sw.d2[at] = d;
          sw.s2[at] = u;
          sw.j2[at] = j;
        }
        n2 += __popc(m);
        __syncwarp();
      }
      // edges to relax: queue 2, or queue 1 itself when the filter is exact
      uint32_t n = shift ? n2 : n1;
      if (n >= 32 || (all && n)) {
        const uint32_t k = min(n, 32u);
        bool want = false;
        uint32_t sd = 0;
        if (lane < k) {
          d = qd[n - k + lane];
          u = qs[n - k + lane];
          j = qj[n - k + lane];
        }
        __syncwarp();
        n -= k;
        if (shift) n2 = n;
        else n1 = n;
        if (lane < k && d != SGS_TOMB) {
          uint32_t su[GMAX], cv[GMAX], cand[GMAX], old[GMAX];
          load_vals<GMAX>(op.val, u, su);
          load_vals<GMAX>(op.val, d, cv);
          sd = g.slots[d];
          uint32_t wt = 1;
          if (g.wmode == W_EXPLICIT) {
            if (op.any_w) wt = H ? *wgt_at(g, g.off[u], j) : g.wgt_d[g.off[u] + j];
          } else if (g.wmode == W_SYNTH) {
            wt = (u + d) % 128u + 1u;
          }
          uint32_t got = 0;
#pragma unroll
          for (int q = 0; q < GMAX; ++q) {
            const bool on_q = (c.lanes >> q & 1u) && (su[q] != INF32 || (op.algo.cc >> q & 1u));
            evald += on_q;
            cand[q] = op.cand_of(su[q] + (op.algo.inc >> q & 1u), wt, q);
            old[q] = 0;
            if (on_q && cand[q] < cv[q]) old[q] = atomicMin(&op.val[(uint64_t)d * GMAX + q], cand[q]);
          }
#pragma unroll
          for (int q = 0; q < GMAX; ++q)
            if (old[q] > cand[q]) {  // strictly lowered
              atomicMin(&op.st[(uint64_t)d * GMAX + q], ((unsigned long long)cand[q] << 32) | u);
              got |= 1u << q;
            }
          want = got && sd && atomicOr(&op.m_out[d], got) == 0u;
        }
        __syncwarp();
        queue.push(out, want, d, sd);
      }
    } while (all ? (n1 | n2) != 0 : n1 >= 32);
  };
  // ---- where windows come from.  Phase 1: `step` consecutive vertices at a
  // time, their blocks' quads one after the other; phase 2, after a grid barrier:
  // slices of the large blocks.  One loop over both, so that the test, the queues
  // and the relaxation are in the code once (inlined at several places they
  // overflowed the instruction cache).
  bool slices = false;                          // phase 2
  uint32_t v0 = 0, ve = 0;                      // vertices of the batch
  uint32_t p = 0, total = 0, s0 = 0;            // positions of the step (phase 2: of the slice)
  uint32_t si = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, ns = 0;  // slice, slices
  uint2 cur = make_uint2(0, 0), nxs = make_uint2(0, 0);
  uint64_t co = 0, nxo = 0;
  uint32_t nxl = 0;
  struct Win {
    uint32_t u, j, left;
    uint4 ids;
  };
  // loads the next window of the positions at hand; false: none is left
  auto fetch = [&](Win &w) -> bool {
    w.left = 0;
    if (p >= total) return false;
    const uint32_t at = p + 4 * lane;
    uint64_t o = co;
    if (slices) {
      w.u = cur.x;
      w.j = cur.y * SWEEP_SLICE + at;
      if (at < total) w.left = total - at;
    } else {
      const uint32_t pe = p + 128u, j = s0 + lane;
      const uint32_t bj = j <= 32u ? sw.eb[j] : total;
      const uint32_t m = __reduce_or_sync(full, (lane && bj < pe) ? 1u << ((bj - p) >> 2) : 0u);
      const uint32_t own = s0 + __popc(m & (full >> (31 - lane)));
      uint32_t nx = s0 + __popc(m);
      if (nx < 32u && sw.eb[nx + 1] <= pe) ++nx;  // an entry starting exactly at pe
      s0 = nx;
      if (at < total) {
        w.u = sw.vtx[own];
        w.j = at - sw.eb[own];
        w.left = sw.len[own] - w.j;
        o = sw.off[own];
      }
    }
    if (w.left) {
      w.ids = ld_quad_stream(H ? adj_at(g, o, w.j) : g.adj_d + o + w.j);
      if constexpr (H)
        if ((o & HOST_BIT) && cache_line(g, (o & OFF_MASK) + w.j) == NO_LINE) host_acc += min(4u, w.left);
    }
    p += 128u;
    return true;
  };
  for (;;) {
    // ---- the next positions
    if (!slices) {
      if (v0 >= ve) {
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(c.next, (unsigned long long)c.batch);
        b = __shfl_sync(full, b, 0);
        if (b >= g.nv) {
          cooperative_groups::this_grid().sync();
          slices = true;
          ns = (uint32_t)__ldcg(c.n_slices);
          if (si < ns) {
            nxs = __ldcg(&c.slices[si]);
            nxl = g.slots[nxs.x];
            nxo = g.off[nxs.x];
          }
          continue;
        }
        v0 = (uint32_t)b;
        ve = (uint32_t)min(b + c.batch, (unsigned long long)g.nv);
      }
      const uint32_t v = v0 + lane;
      uint32_t len = lane < c.step && v < ve ? g.slots[v] : 0u;
      v0 += c.step;
      uint64_t o = 0;
      if (len) {
        uint32_t x[GMAX];
        load_vals<GMAX>(op.val, v, x);
        o = g.off[v];
        const uint32_t l = g.live[v];
        uint32_t m = 0;
#pragma unroll
        for (int q = 0; q < GMAX; ++q) {
          const bool r = (c.lanes >> q & 1u) && (x[q] != INF32 || (op.algo.cc >> q & 1u));
          m |= (r ? 1u : 0u) << q;
          edges[q] += r ? l : 0u;
        }
        if (!m) len = 0;
        else walked += (1ull << CNT_SHIFT) | ((len + 3u) & ~3u);
        if constexpr (H) {
          if (len && (o & HOST_BIT)) {
            hot_bump(g, v, o);
            host_all += len;
            o = resolve_block(g, o, len);
          }
        }
      }
      // slices of large blocks
      for (uint32_t big = __ballot_sync(full, len > SWEEP_BIG); big; big &= big - 1) {
        const int from = __ffs(big) - 1;
        const uint32_t n = (__shfl_sync(full, len, from) + SWEEP_SLICE - 1) / SWEEP_SLICE;
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(c.n_slices, (unsigned long long)n);
        at = __shfl_sync(full, at, 0);
        const uint32_t bv = __shfl_sync(full, v, from);
        for (uint32_t i = lane; i < n; i += 32) c.slices[at + i] = make_uint2(bv, i);
      }
      if (len > SWEEP_BIG) len = 0;
      const uint32_t some = __ballot_sync(full, len != 0u);
      if (!some) continue;
      const uint32_t pad = (len + 3u) & ~3u;
      uint32_t x = pad;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(full, x, d);
        if (lane >= (uint32_t)d) x += y;
      }
      total = __shfl_sync(full, x, 31);
      const uint32_t ne = __popc(some);
      __syncwarp();  // the last step's entries are read
      if (lane >= ne) sw.eb[lane] = total;
      if (lane == 0) sw.eb[32] = total;
      if (len) {
        const uint32_t at = __popc(some & below);
        sw.eb[at] = x - pad;
        sw.off[at] = o;
        sw.len[at] = len;
        sw.vtx[at] = v;
      }
      __syncwarp();
      s0 = 0;
    } else {
      if (si >= ns) break;
      cur = nxs;
      co = nxo;
      total = min(nxl - cur.y * SWEEP_SLICE, SWEEP_SLICE);
      si += gridDim.x * (SWEEP_THREADS / 32);
      if (si < ns) {  // the next slice's place, while this one is walked
        nxs = __ldcg(&c.slices[si]);
        nxl = g.slots[nxs.x];
        nxo = g.off[nxs.x];
      }
    }
    p = 0;
    // ---- its windows, two in flight ahead of the one tested
    Win wa{}, wb{};
    bool more = fetch(wa), more_b = fetch(wb);
#pragma unroll 1
    while (more) {
      Win wc{};
      const bool more_c = fetch(wc);
      uint32_t hit = 0;
      if (wa.left) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t d = quad_at(wa.ids, k);
          hit |= (__funnelshift_r(filter[d >> shift5 & mask], 0u, d >> shift) & 1u) << k;
        }
        hit &= wa.left >= 4u ? 0xFu : (1u << wa.left) - 1u;
      }
      // the hits into queue 1: all together where they fit, else quad slot by
      // quad slot
      const uint32_t nh = __popc(hit);
      const uint32_t h0 = __ballot_sync(full, nh & 1u), h1 = __ballot_sync(full, nh & 2u);
      uint32_t ks = 0;
      const uint32_t all = __popc(h0) + 2 * __popc(h1);  // (a lane with four hits counts none here)
      if (__any_sync(full, nh == 4u) || all > 32u) {
        ks = __reduce_or_sync(full, hit);
      } else if (all) {
        uint32_t at = n1 + __popc(h0 & below) + 2 * __popc(h1 & below);
        for (uint32_t h = hit; h; h &= h - 1) {
          const int k = __ffs(h) - 1;
          sw.d1[at] = quad_at(wa.ids, k);
          sw.s1[at] = wa.u;
          sw.j1[at] = wa.j + k;
          ++at;
        }
        n1 += all;
        __syncwarp();
        if (n1 >= 32) drain(false);
      }
#pragma unroll 1
      while (ks) {
        const int k = __ffs(ks) - 1;
        ks &= ks - 1;
        const bool h = hit >> k & 1u;
        const uint32_t m = __ballot_sync(full, h);
        if (h) {
          const uint32_t at = n1 + __popc(m & below);
          sw.d1[at] = quad_at(wa.ids, k);
          sw.s1[at] = wa.u;
          sw.j1[at] = wa.j + k;
        }
        n1 += __popc(m);
        __syncwarp();
        if (n1 >= 32) drain(false);
      }
      wa = wb;
      wb = wc;
      more = more_b;
      more_b = more_c;
    }
  }
  if (n1 | n2) drain(true);
  queue.template finish<SWEEP_THREADS>(out);
  // ---- counts: one atomic per CTA and counter
  __syncthreads();  // the filter is done with; its first words hold the sums
  unsigned long long *sum = reinterpret_cast<unsigned long long *>(filter);
  constexpr int NS = GMAX + 4;
  if (threadIdx.x < NS) sum[threadIdx.x] = 0;
  __syncthreads();
  auto add = [&](int k, unsigned long long x) {
    x = warp_sum(x);
    if (lane == 0 && x) atomicAdd(&sum[k], x);
  };
#pragma unroll
  for (int q = 0; q < GMAX; ++q) add(q, edges[q]);
  add(GMAX, walked);
  add(GMAX + 1, evald);
  if constexpr (H) {
    add(GMAX + 2, host_acc);
    add(GMAX + 3, host_all);
  }
  __syncthreads();
  if (threadIdx.x < NS && sum[threadIdx.x]) {
    const unsigned long long x = sum[threadIdx.x];
    const int k = threadIdx.x;
    if (k < GMAX) atomicAdd(&c.lane_edges[k], x);
    else if (k == GMAX) atomicAdd(c.walked, x);
    else if (k == GMAX + 1) atomicAdd(c.edge_stat, x);
    else if (k == GMAX + 2) atomicAdd(c.host_stat, x);
    if (k == GMAX + 2 && g.cstat) atomicAdd(&g.cstat[1], x);
    if (k == GMAX + 3 && g.cstat) atomicAdd(&g.cstat[0], x);
  }
}

// One vertex, given lanes (the source of new BFS/SSSP lanes).
__global__ void k_group_seed_one(GraphView g, uint32_t v, uint32_t bits, uint32_t *m_out,
                                 FrontierView out) {
  if (threadIdx.x >= 32) return;
  const uint32_t d = g.slots[v];
  bool want = false;
  if (threadIdx.x == 0 && d) want = atomicOr(&m_out[v], bits) == 0u;
  frontier_append(out, want, v, d);
}

// Deletion seeds: deleted (u,v) whose lane-q parent of v is u reset lane q.
template <int S>
__global__ void k_group_seed_deleted(GraphView g, unsigned long long *st, uint32_t *val, uint32_t lanes,
                                     LaneAlgo algo, const uint64_t *keys, uint32_t n,
                                     unsigned long long *inval, uint32_t *mark, uint32_t *m_out,
                                     FrontierView out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  __shared__ uint32_t s_reset[S];
  if (threadIdx.x < S) s_reset[threadIdx.x] = 0;
  __syncthreads();
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < n; b += stride) {
    const uint64_t i = b + threadIdx.x;
    bool want = false;
    uint32_t v = 0, d = 0;
    if (i < n) {
      const uint64_t k = keys[i];
      const uint32_t u = (uint32_t)(k >> 32);
      v = (uint32_t)k;
      uint32_t bits = 0;
      unsigned long long row[S], was[S];
      load_row<S>(st, v, row);
      d = g.slots[v];
#pragma unroll
      for (int q = 0; q < S; ++q) {
        was[q] = ~row[q];
        if ((lanes >> q & 1u) && (uint32_t)row[q] == u)
          was[q] = atomicCAS(&st[(uint64_t)v * S + q], row[q],
                             algo.at(q) == A_CC ? (((unsigned long long)v << 32) | INF32) : ~0ull);
      }
#pragma unroll
      for (int q = 0; q < S; ++q) {
        if (was[q] != row[q]) continue;
        val[(uint64_t)v * S + q] = algo.at(q) == A_CC ? v : INF32;
        bits |= 1u << q;
        atomicAdd(&s_reset[q], 1u);
      }
      if (bits) {
        if (mark) bit_set(mark, v);
        want = d && atomicOr(&m_out[v], bits) == 0u;
      }
    }
    frontier_append_block(out, want, v, d);
  }
  __syncthreads();
  if (threadIdx.x < S && s_reset[threadIdx.x])
    atomicAdd(&inval[threadIdx.x], (unsigned long long)s_reset[threadIdx.x]);
}

// Relaxes just the kept inserted edges in the selected lanes: the whole
// repair of an insert-only batch, and the inserted-edge half of the repair
// after an invalidation (the other half is the restricted first round).
// With `resets` the repair's mode decides: FULL, nothing (the full sweep
// covers the inserted edges); RESTRICTED, improved vertices go to frontier 1
// (out1, m_out1) and the edges are not counted (the sweep's count has them);
// NONE, to frontier 0 (out, m_out).
template <int S>
__global__ void k_group_relax_inserted(GraphView g, unsigned long long *st, uint32_t *val, uint32_t lanes,
                                       LaneAlgo algo, const uint64_t *keys, const uint32_t *w,
                                       const uint32_t *n_ptr, uint32_t *m_out, FrontierView out,
                                       unsigned long long *lane_edges,
                                       const unsigned long long *resets = nullptr,
                                       unsigned long long restrict_max = 0, uint32_t *m_out1 = nullptr,
                                       FrontierView out1 = FrontierView{}) {
  if (resets) {
    const int mode = repair_mode(resets, lanes, restrict_max);
    if (mode == REPAIR_FULL) return;
    if (mode == REPAIR_RESTRICTED) {
      out = out1;
      m_out = m_out1;
      lane_edges = nullptr;
    }
  }
  const uint32_t n = *n_ptr;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint32_t counted = 0;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < n; b += stride) {
    const uint64_t i = b + threadIdx.x;
    bool want = false;
    uint32_t v = 0, d = 0;
    if (i < n) {
      const uint64_t k = keys[i];
      const uint32_t u = (uint32_t)(k >> 32);
      v = (uint32_t)k;
      ++counted;
      uint32_t su[S], sv[S];
      load_vals<S>(val, u, su);
      load_vals<S>(val, v, sv);
      uint32_t bits = 0, cand[S], old[S];
      d = g.slots[v];
      const uint32_t wi = g.wmode == W_EXPLICIT ? (w ? w[i] : 1u) : g.wmode == W_SYNTH ? (u + v) % 128u + 1u : 1u;
#pragma unroll
      for (int q = 0; q < S; ++q) {
        const int a = algo.at(q);
        uint64_t nd = su[q];
        if (a != A_CC) nd += a == A_SSSP ? wi : 1u;
        const bool ok = (lanes >> q & 1u) && (a == A_CC || su[q] != INF32) && nd < sv[q];
        cand[q] = (uint32_t)nd;
        old[q] = 0;
        if (ok) old[q] = atomicMin(&val[(uint64_t)v * S + q], cand[q]);
      }
#pragma unroll
      for (int q = 0; q < S; ++q)
        if (old[q] > cand[q]) {  // strictly lowered
          atomicMin(&st[(uint64_t)v * S + q], ((unsigned long long)cand[q] << 32) | u);
          bits |= 1u << q;
        }
      if (bits) want = d && atomicOr(&m_out[v], bits) == 0u;
    }
    frontier_append_block(out, want, v, d);
  }
  if (!lane_edges) return;
  // one atomic per CTA and lane
  __shared__ uint32_t s_count;
  if (threadIdx.x == 0) s_count = 0;
  __syncthreads();
  counted = warp_sum(counted);
  if ((threadIdx.x & 31) == 0 && counted) atomicAdd(&s_count, counted);
  __syncthreads();
  if (threadIdx.x < S && (lanes >> threadIdx.x & 1u) && s_count)
    atomicAdd(&lane_edges[threadIdx.x], (unsigned long long)s_count);
}

// One lane of every vertex: its values from the mirror (between snapshots
// equal to the packed words' values, and half their bytes per row), or with
// val == null its parents from the packed words.  Bound by the rows' sectors:
// a lane's 4 or 8 bytes cost a 32-B sector each, which narrow values share
// between two vertices.
template <int S>
__global__ void k_group_column(const unsigned long long *st, const uint32_t *val, uint32_t nv, int lane,
                               uint32_t *out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride)
    out[v] = val ? val[v * S + lane] : (uint32_t)st[v * S + lane];
}

template <int S>
__global__ void k_group_summary(const unsigned long long *st, uint32_t nv, int lane,
                                unsigned long long *out) {
  unsigned long long reached = 0, sum = 0, mx = 0, psum = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride) {
    const unsigned long long s = st[v * S + lane];
    const uint32_t val = (uint32_t)(s >> 32);
    if (val == INF32) continue;
    reached += 1;
    sum += val;
    mx = val > mx ? val : mx;
    if ((uint32_t)s != INF32) psum += (uint32_t)s;
  }
  reached = warp_sum(reached);
  sum = warp_sum(sum);
  psum = warp_sum(psum);
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, mx, s);
    mx = o > mx ? o : mx;
  }
  if ((threadIdx.x & 31) == 0) {
    if (reached) atomicAdd(&out[0], reached);
    if (sum) atomicAdd(&out[1], sum);
    atomicMax(&out[2], mx);
    if (psum) atomicAdd(&out[3], psum);
  }
}

// The same summaries for several lanes of a narrow group in one pass over
// the state rows (one 32-B row per vertex read once for all of them):
// slot[q] >= 0 selects lane q and its 4 counters at out + 4 * slot[q].
struct LaneSlots {
  int slot[GMAX];
};
__global__ void k_group_summary_lanes(const unsigned long long *st, uint32_t nv, LaneSlots ls,
                                      unsigned long long *out) {
  unsigned long long reached[GMAX] = {}, sum[GMAX] = {}, mx[GMAX] = {}, psum[GMAX] = {};
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride) {
    const ulonglong2 a = __ldcs(reinterpret_cast<const ulonglong2 *>(st + v * GMAX));
    const ulonglong2 b = __ldcs(reinterpret_cast<const ulonglong2 *>(st + v * GMAX + 2));
    const unsigned long long row[GMAX] = {a.x, a.y, b.x, b.y};
#pragma unroll
    for (int q = 0; q < GMAX; ++q) {
      if (ls.slot[q] < 0) continue;
      const uint32_t val = (uint32_t)(row[q] >> 32);
      if (val == INF32) continue;
      reached[q] += 1;
      sum[q] += val;
      mx[q] = val > mx[q] ? val : mx[q];
      if ((uint32_t)row[q] != INF32) psum[q] += (uint32_t)row[q];
    }
  }
#pragma unroll
  for (int q = 0; q < GMAX; ++q) {
    if (ls.slot[q] < 0) continue;
    const unsigned long long r = warp_sum(reached[q]), su = warp_sum(sum[q]), ps = warp_sum(psum[q]);
    unsigned long long m = mx[q];
#pragma unroll
    for (int sh = 16; sh > 0; sh >>= 1) {
      const unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, m, sh);
      m = o > m ? o : m;
    }
    if ((threadIdx.x & 31) == 0) {
      unsigned long long *o = out + 4 * ls.slot[q];
      if (r) atomicAdd(&o[0], r);
      if (su) atomicAdd(&o[1], su);
      atomicMax(&o[2], m);
      if (ps) atomicAdd(&o[3], ps);
    }
  }
}

// Lanes present in a frontier: the OR of its entries' masks (narrow u32 or wide
// u64), for a serving loop that retires a lane as soon as no entry carries it.
template <class M>
__global__ void k_lanes_present(const uint32_t *vtx, const unsigned long long *cnt, const M *mask,
                                unsigned long long *out) {
  const uint32_t n = (uint32_t)(__ldcg(cnt) >> CNT_SHIFT);
  unsigned long long m = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    m |= (unsigned long long)__ldcg(&mask[__ldcg(&vtx[i])]);
  const uint32_t lo = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)m);
  const uint32_t hi = sizeof(M) == 8 ? __reduce_or_sync(0xFFFFFFFFu, (uint32_t)(m >> 32)) : 0u;
  if ((threadIdx.x & 31) == 0 && (lo | hi)) atomicOr(out, (unsigned long long)hi << 32 | lo);
}

// Dense seeding of CC lanes into a frontier that may already hold entries:
// OR the lanes in, append only vertices whose mask was empty.
template <class M>
__global__ void k_seed_all_or(GraphView g, M bits, M *m_out, FrontierView out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < g.nv; b += stride) {
    const uint64_t v = b + threadIdx.x;
    bool want = false;
    uint32_t d = 0;
    if (v < g.nv) {
      d = g.slots[v];
      if (d) want = atomicOr(&m_out[v], bits) == (M)0;
    }
    frontier_append_block(out, want, (uint32_t)v, d);
  }
}

// Masks of the last non-empty frontier (after convergence).
__global__ void k_clear_masks(const uint32_t *vtx, const unsigned long long *cnt, uint32_t *mask) {
  clear_prev_masks(vtx, cnt, mask);
}

}  // namespace sgs
