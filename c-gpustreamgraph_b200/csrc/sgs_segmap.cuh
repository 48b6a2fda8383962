// sgs_segmap.cuh -- the engine's load-balanced segmented map kernel
// (template only, so several translation units can instantiate it).
#pragma once
#include <cub/block/block_reduce.cuh>
#include <type_traits>
#include <utility>

#include "sgs_device.cuh"

namespace sgs {

// ---------------------------------------------------------------------------
// Generic load-balanced segmented map.
//
// The input frontier is a list of entries (vertex v, ebase) whose ranges
// [ebase_s, ebase_{s+1}) tile [0, T).  Units of UNIT consecutive positions are
// spread over a fixed grid; a CTA stages up to CHUNK entries of its unit in
// shared memory (the per-entry payload is loaded once, coalesced) and then
// its threads walk consecutive positions, so consecutive lanes touch
// consecutive slots of the same block (coalesced 128-B lines).  Every thread
// of a CTA runs the same trip count, so warp-aggregated appends always see
// full warps.
// ---------------------------------------------------------------------------
constexpr int CHUNK = 256;

// Ops that define touch(v, payload) are told once per frontier entry (by the
// CTA that owns the entry's first slot); PageRank's push counts hotness there.
template <class Op, class = void>
struct op_touches : std::false_type {};
template <class Op>
struct op_touches<Op, std::void_t<decltype(std::declval<const Op &>().touch(
                          0u, std::declval<const typename Op::Payload &>()))>> : std::true_type {};

// Ops either implement visit (one slot) or, with kQuad, visit4 (four
// consecutive slots j0..j0+3 of one block, j0 a multiple of 4; slots >= len
// are padding and must be ignored).
template <class Op>
__device__ __forceinline__ uint32_t visit_quad(const Op &op, uint32_t u,
                                               const typename Op::Payload &p, uint32_t j0,
                                               uint32_t len, bool (&app)[4], uint32_t (&av)[4],
                                               uint32_t (&ad)[4]) {
  if constexpr (Op::kQuad) {
    return op.visit4(u, p, j0, len, app, av, ad);
  } else {
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (j0 + k < len) c += op.visit(u, p, j0 + k, app[k], av[k], ad[k]);
    return c;
  }
}

// A warp's walk over its share of a staged chunk, one window of 32 quads (128
// positions) per step, lane i on quad i.  Owners need no search per quad: lane
// j holds the start of entry s0 + j (s0 = owner of the window's first quad),
// every start inside the window sets bit (start - window) / 4 of a warp-wide
// OR, and a lane's owner is s0 plus the set bits at or below its quad.  The
// entries of the chunk must all have slots: a window then meets at most 32 of
// them and no two starts share a bit.  The same bits give the next window's
// first owner.  (With a binary search per quad, eight dependent shared-memory
// reads, tombstoning 500,000 deletes at scale 24 took 420 us instead of 402.)
// A chunk with an empty entry, which none of the engine's frontiers has, is
// walked by that search.
template <int GC>
struct WindowWalk {
  const uint64_t *eb;   // [GC + 1] starts of the chunk's entries
  const uint32_t *len;  // [GC] their slots
  uint64_t q, end;      // this warp's share in quads: next window, end
  int s0;
  // Warp `wid` of `nw`, over positions [lo, hi) of the chunk.
  __device__ __forceinline__ WindowWalk(const uint64_t *eb_, const uint32_t *len_, uint64_t lo, uint64_t hi,
                                        uint32_t wid, uint32_t nw)
      : eb(eb_), len(len_) {
    const uint64_t nq = hi > lo ? (hi - lo) >> 2 : 0;
    q = (lo >> 2) + nq * wid / nw;
    end = (lo >> 2) + nq * (wid + 1) / nw;
    int a = 0, b = GC - 1;
    if (q < end)
      while (a < b) {  // owner of the share's first quad, once per chunk
        const int m = (a + b + 1) >> 1;
        if (eb[m] <= q << 2) a = m;
        else b = m - 1;
      }
    s0 = a;
  }
  // The window at q: this lane's owner and its first slot there; true when
  // the quad holds slots.  All 32 lanes, while q < end; moves on by a window.
  __device__ __forceinline__ bool next(int &own, uint32_t &j0) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t p0 = q << 2, pe = p0 + 4 * 32;
    const int j = s0 + (int)lane;
    const uint64_t bj = j <= GC ? eb[j] : ~0ull;
    const uint32_t bit = (lane >= 1 && bj < pe) ? 1u << (uint32_t)((bj - p0) >> 2) : 0u;
    const uint32_t m = __reduce_or_sync(0xFFFFFFFFu, bit);
    own = s0 + __popc(m & (0xFFFFFFFFu >> (31 - lane)));
    int ns = s0 + __popc(m);
    if (ns < GC && eb[ns + 1] <= pe) ++ns;  // an entry starting exactly at pe
    s0 = ns;
    const bool in = q + lane < end && own < GC;
    j0 = in ? (uint32_t)(p0 + 4 * lane - eb[own]) : 0u;
    q += 32;
    return in && j0 < len[own];
  }
  // The same where entries may be empty: the last that starts at or before the
  // quad, which is the one with slots.
  __device__ __forceinline__ bool search(int &own, uint32_t &j0) {
    const uint64_t p = (q + (threadIdx.x & 31)) << 2;
    const bool in = q + (threadIdx.x & 31) < end;
    int a = 0, b = GC - 1;
    while (in && a < b) {
      const int m = (a + b + 1) >> 1;
      if (eb[m] <= p) a = m;
      else b = m - 1;
    }
    own = a;
    j0 = in ? (uint32_t)(p - eb[a]) : 0u;
    q += 32;
    return in && j0 < len[a];
  }
};

// Each CTA walks one contiguous run of units [u_begin, u_end), staging up to
// CHUNK entries at a time in shared memory; its warps share the chunk's
// positions, each thread on four consecutive ones per step.
template <class Op>
__global__ void __launch_bounds__(RELAX_THREADS)
    seg_map(FrontierView in, FrontierView out, Op op, unsigned long long *edge_stat) {
  using P = typename Op::Payload;
  __shared__ uint64_t s_eb[CHUNK + 1];
  __shared__ uint32_t s_len[CHUNK];
  __shared__ P s_pay[CHUNK];
  __shared__ uint32_t s_vtx[CHUNK];
  const uint64_t packed = __ldcg((const unsigned long long *)in.counter);
  const uint32_t n = (uint32_t)(packed >> CNT_SHIFT);
  const uint64_t T = packed & EDGE_MASK;
  uint64_t counted = 0;
  const uint64_t nunits = (T + UNIT - 1) / UNIT;
  const uint64_t ub = (uint64_t)blockIdx.x * nunits / gridDim.x;
  const uint64_t ue = (uint64_t)(blockIdx.x + 1) * nunits / gridDim.x;
  if (n != 0 && ub < ue) {
    const uint64_t E0 = ub * UNIT;
    const uint64_t E1 = min(ue * (uint64_t)UNIT, T);
    uint32_t s = __ldcg(&in.ustart[ub]);
    for (;;) {
      __syncthreads();  // previous chunk fully consumed
      bool empty = false;
      {
        const uint32_t t = threadIdx.x;
        const uint32_t idx = s + t;
        const uint64_t eb = idx < n ? __ldcg((const unsigned long long *)&in.ebase[idx]) : T;
        s_eb[t] = eb;
        if (t == 0) {
          const uint32_t j = s + CHUNK;
          s_eb[CHUNK] = j < n ? __ldcg((const unsigned long long *)&in.ebase[j]) : T;
        }
        if (idx < n && eb < E1) {
          const uint32_t v = __ldcg(&in.vtx[idx]);
          s_vtx[t] = v;
          const uint32_t len = __ldcg(&in.len[idx]);
          s_len[t] = len;
          empty = len == 0;
          s_pay[t] = op.load(idx, v);
          if constexpr (op_touches<Op>::value)
            if (eb >= E0) op.touch(v, s_pay[t]);
        }
      }
      const bool any_empty = __syncthreads_or(empty);
      const uint64_t lo = max(E0, s_eb[0]);
      const uint64_t hi = min(E1, s_eb[CHUNK]);
      WindowWalk<CHUNK> walk(s_eb, s_len, lo, hi, threadIdx.x >> 5, RELAX_THREADS / 32);
      while (walk.q < walk.end) {
        bool app[4] = {false, false, false, false};
        uint32_t av[4] = {0, 0, 0, 0}, ad[4] = {0, 0, 0, 0};
        int l;
        uint32_t j0;
        if (any_empty ? walk.search(l, j0) : walk.next(l, j0)) counted += visit_quad(op, s_vtx[l], s_pay[l], j0, s_len[l], app, av, ad);
        if (Op::kAppends) {
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) frontier_append(out, app[k], av[k], ad[k]);
        }
      }
      if (s_eb[CHUNK] >= E1 || s + CHUNK >= n) break;
      s += CHUNK;
    }
  }
  if (edge_stat) {
    typedef cub::BlockReduce<unsigned long long, RELAX_THREADS> BR;
    __shared__ typename BR::TempStorage tmp;
    unsigned long long tot = BR(tmp).Sum((unsigned long long)counted);
    if (threadIdx.x == 0 && tot) atomicAdd(edge_stat, tot);
  }
}

}  // namespace sgs
