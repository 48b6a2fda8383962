// sgs_kernels.cuh -- sm_100a kernels of the streaming-graph engine.
//
// Reference behaviour each kernel re-implements (paths relative to the
// reference project):
//   seg_map (sgs_segmap.cuh) and the group ops (sgs_group.cuh)
//                         <- kernel::SyncPushDDBDelta / RelaxCTADB /
//                            CTAWorkSchedulerNew / PushFunctorDB
//                            (variants/driver.cuh:1893-1935,
//                             variants/sync_push_dd.cuh:170-268,
//                             groute/device/cta_scheduler_hybrid.cuh:59-245,
//                             variants/push_functor.h:252-321), the deletion
//                            phase reset_del_edges + SyncPushDDB_del
//                            (driver.cuh:398-430, :1985-2031) and the
//                            all-vertices re-push SyncPushDDBAll (:1727-1761)
//   frontier_append       <- RebuildWorklist* + dev::Queue::append
//                            (driver.cuh:654-909, groute/device/queue.cuh:84-88)
//   PR absorb/push/amend  <- hybrid_pr.cu:66-122 CombineValueBuffer /
//                            CombineValueBufferAmend / AccumulateBuffer and
//                            SyncPushDDBAmend (driver.cuh:1770-1804)
//   batch-apply kernels   <- host::PMAGraph::insert / del_edge
//                            (groute/graphs/csr_graph.cuh:658-811), done on
//                            the device as sort + tombstone + append/relocate
#pragma once
#include <cub/block/block_reduce.cuh>

#include "sgs_device.cuh"
#include "sgs_segmap.cuh"
#include "sgs_steplen.cuh"

namespace sgs {

// ---------------------------------------------------------------------------
// Ops
// ---------------------------------------------------------------------------
// PageRank push of a per-source scalar (absorbed residual or +-alpha*x/deg).
struct PrPay {
  uint64_t off;
  double c;
};
struct PrPushOp {
  static constexpr bool kAppends = false;
  static constexpr bool kQuad = true;
  using Payload = PrPay;
  GraphView g;
  const double *pv;   // per-vertex push value (alpha * r / outdeg)
  double *r;
  __device__ __forceinline__ Payload load(uint32_t, uint32_t v) const {
    PrPay p;
    p.off = g.off[v];
    p.c = pv[v];
    return p;
  }
  __device__ __forceinline__ void touch(uint32_t v, const Payload &p) const { hot_bump(g, v, p.off); }
  __device__ __forceinline__ uint32_t visit(uint32_t, const Payload &p, uint32_t j,
                                            bool &, uint32_t &, uint32_t &) const {
    const uint32_t dst = *adj_at(g, p.off, j);
    if (dst == SGS_TOMB) return 0;
    if (p.c != 0.0) atomicAdd(&r[dst], p.c);
    return 1;
  }
  __device__ __forceinline__ uint32_t visit4(uint32_t, const Payload &p, uint32_t j0, uint32_t len,
                                             bool (&)[4], uint32_t (&)[4], uint32_t (&)[4]) const {
    const uint4 ids = ld_quad(adj_at(g, p.off, j0));
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t dst = quad_at(ids, k);
      if (j0 + k >= len || dst == SGS_TOMB) continue;
      ++c;
      if (p.c != 0.0) atomicAdd(&r[dst], p.c);
    }
    return c;
  }
};
// Cancel (sign=-1, old graph) / compensate (sign=+1, new graph) of
// hybrid_pr.cu:88-106, restricted to sources whose out-edges changed.
struct PrAmendOp {
  static constexpr bool kAppends = false;
  static constexpr bool kQuad = false;
  using Payload = PrPay;
  GraphView g;
  const double *x;
  double *r;
  double scale;  // sign * alpha
  __device__ __forceinline__ Payload load(uint32_t, uint32_t v) const {
    PrPay p;
    p.off = g.off[v];
    const uint32_t l = g.live[v];
    p.c = l ? scale * x[v] / (double)l : 0.0;
    return p;
  }
  __device__ __forceinline__ uint32_t visit(uint32_t, const Payload &p, uint32_t j,
                                            bool &, uint32_t &, uint32_t &) const {
    const uint32_t dst = *adj_at(g, p.off, j);
    if (dst == SGS_TOMB) return 0;
    if (p.c != 0.0) atomicAdd(&r[dst], p.c);
    return 1;
  }
};

// Tombstone every slot of u whose destination is in u's sorted delete group
// (PMAGraph::del_edge removes every matching entry).  Four slots per thread,
// each looked up by binary search in the group (a few L1-resident lines); the
// block is read with a plain (coherent) load because this kernel writes it.
struct GroupPay {
  uint64_t off;
  uint32_t gs, ge;
};
struct TombOp {
  static constexpr bool kAppends = false;
  static constexpr bool kQuad = true;
  using Payload = GroupPay;
  GraphView g;
  const uint64_t *keys;   // sorted delete keys (src<<32|dst)
  const uint32_t *gstart; // per entry
  uint32_t nkeys;
  __device__ __forceinline__ Payload load(uint32_t slot, uint32_t v) const {
    GroupPay p;
    p.off = g.off[v];
    p.gs = gstart[slot];
    // end of the group: first key with a larger source.  Galloping from
    // the group start: most sources have one or two deletes, so the first
    // probe usually ends it; a hub's long group takes log2(size) probes.
    const uint64_t lim = ((uint64_t)v + 1) << 32;
    uint32_t lo = p.gs + 1, step = 1, hi = p.gs + 1;  // keys[gs] < lim
    while (hi < nkeys && keys[hi] < lim) {
      lo = hi + 1;
      step <<= 1;
      hi = p.gs + step;
    }
    uint32_t r = hi < nkeys ? hi : nkeys;
    uint32_t l = lo;
    while (l < r) {
      const uint32_t m = (l + r) >> 1;
      if (keys[m] < lim) l = m + 1;
      else r = m;
    }
    p.ge = l;
    return p;
  }
  __device__ __forceinline__ uint32_t visit(uint32_t, const Payload &, uint32_t, bool &, uint32_t &,
                                            uint32_t &) const {
    return 0;
  }
  __device__ __forceinline__ uint32_t visit4(uint32_t u, const Payload &p, uint32_t j0, uint32_t len,
                                             bool (&)[4], uint32_t (&)[4], uint32_t (&)[4]) const {
    uint32_t *a = adj_wptr(g, p.off) + j0;
    uint32_t *ca = cache_slot_w(g, g.adj_c, p.off, j0);  // cached copy: read from it, write both
    const uint4 q = *reinterpret_cast<const uint4 *>(ca ? ca : a);
    uint64_t key[4];
    bool ok[4];
    bool any = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t dst = quad_at(q, k);
      ok[k] = j0 + k < len && dst != SGS_TOMB;
      key[k] = ((uint64_t)u << 32) | dst;
      any |= ok[k];
    }
    if (!any) return 0;
    // the four lower bounds in lockstep (branchless, the same trip count for
    // all: it depends only on the group's length), so their dependent loads
    // overlap instead of running one search after the other
    uint32_t lo[4] = {p.gs, p.gs, p.gs, p.gs};
    uint32_t n = p.ge - p.gs;  // >= 1: the entry has deletes
    while (n > 1) {
      const uint32_t half = n >> 1;
#pragma unroll
      for (int k = 0; k < 4; ++k) lo[k] = __ldg(&keys[lo[k] + half]) < key[k] ? lo[k] + half : lo[k];
      n -= half;
    }
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (!ok[k]) continue;
      const uint64_t kk = __ldg(&keys[lo[k]]);
      const uint32_t at = kk < key[k] ? lo[k] + 1 : lo[k];
      if (at < p.ge && (at == lo[k] ? kk : __ldg(&keys[at])) == key[k]) {
        a[k] = SGS_TOMB;
        if (ca) ca[k] = SGS_TOMB;
        ++c;
      }
    }
    if (c) atomicSub(&g.live[u], c);
    return c;
  }
};

// Copy of a whole block (slots as they are, tombstones included) from an old
// location to the vertex's current block; used by relocation and repacking.
struct CopyPay {
  uint64_t from;
  uint64_t to;
};
struct CopyBlockOp {
  static constexpr bool kAppends = false;
  static constexpr bool kQuad = false;
  using Payload = CopyPay;
  GraphView g;
  const uint64_t *from_off;  // per vertex: old offset (tier bit included)
  const uint64_t *to_off;    // per vertex: new offset
  uint32_t *src_adj_d, *src_wgt_d, *src_adj_h, *src_wgt_h;  // source arenas
  __device__ __forceinline__ Payload load(uint32_t, uint32_t v) const {
    CopyPay p;
    p.from = from_off[v];
    p.to = to_off[v];
    return p;
  }
  __device__ __forceinline__ uint32_t visit(uint32_t, const Payload &p, uint32_t j,
                                            bool &, uint32_t &, uint32_t &) const {
    const uint64_t fo = p.from & OFF_MASK;
    const bool fh = (p.from & HOST_BIT) != 0;
    const uint32_t a = (fh ? src_adj_h : src_adj_d)[fo + j];
    adj_wptr(g, p.to)[j] = a;
    if (g.wmode == W_EXPLICIT) wgt_wptr(g, p.to)[j] = (fh ? src_wgt_h : src_wgt_d)[fo + j];
    return 0;
  }
};

// Copy an input CSR (device arrays) into the arena blocks.
struct LoadCsrOp {
  static constexpr bool kAppends = false;
  static constexpr bool kQuad = false;
  using Payload = CopyPay;
  GraphView g;
  const uint64_t *row;
  const uint32_t *col;
  const uint32_t *w;   // null unless weights are explicit
  __device__ __forceinline__ Payload load(uint32_t, uint32_t v) const {
    CopyPay p;
    p.from = row[v];
    p.to = g.off[v];
    return p;
  }
  __device__ __forceinline__ uint32_t visit(uint32_t, const Payload &p, uint32_t j,
                                            bool &, uint32_t &, uint32_t &) const {
    adj_wptr(g, p.to)[j] = col[p.from + j];
    if (w) wgt_wptr(g, p.to)[j] = w[p.from + j];
    return 0;
  }
};

// Export blocks (live edges only) into a CSR whose row offsets are given.  A
// block without tombstones keeps its order; otherwise live slots are placed
// through a per-vertex counter (order not kept).
struct ExportPay {
  uint64_t from;
  uint64_t to;
  uint32_t dense;
  uint32_t pad;
};
struct ExportOp {
  static constexpr bool kAppends = false;
  static constexpr bool kQuad = false;
  using Payload = ExportPay;
  GraphView g;
  const uint64_t *row_out;
  uint32_t *col_out;
  uint32_t *w_out;
  uint32_t *fill;  // per-vertex fill counter (zeroed)
  __device__ __forceinline__ Payload load(uint32_t, uint32_t v) const {
    ExportPay p;
    p.from = g.off[v];
    p.to = row_out[v];
    p.dense = g.slots[v] == g.live[v];
    p.pad = 0;
    return p;
  }
  __device__ __forceinline__ uint32_t visit(uint32_t u, const Payload &p, uint32_t j,
                                            bool &, uint32_t &, uint32_t &) const {
    const uint32_t dst = adj_ptr(g, p.from)[j];
    if (dst == SGS_TOMB) return 0;
    const uint32_t k = p.dense ? j : atomicAdd(&fill[u], 1u);
    col_out[p.to + k] = dst;
    if (w_out) w_out[p.to + k] = edge_weight(g, p.from, j, u, dst);
    return 1;
  }
};

// ---------------------------------------------------------------------------
// Frontier builders (all lanes of every warp reach frontier_append)
// ---------------------------------------------------------------------------
__global__ void k_append_one(FrontierView out, uint32_t v, uint32_t d) {
  if (threadIdx.x >= 32) return;
  frontier_append(out, threadIdx.x == 0 && d > 0, v, d);
}

// Every vertex with a non-empty block (PageRank rounds, loads, repacks).
__global__ void k_dense_frontier(GraphView g, FrontierView out) {
  constexpr int N = 8;  // consecutive vertices per thread, one block append per 2048
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * N;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x * N; b < g.nv; b += stride) {
    const uint64_t v0 = b + (uint64_t)threadIdx.x * N;
    bool want[N];
    uint32_t d[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      d[i] = v0 + i < g.nv ? g.slots[v0 + i] : 0u;
      want[i] = d[i] > 0;
    }
    frontier_append_block_n<N>(out, want, (uint32_t)v0, d);
  }
}

// PageRank: value 0, buffer (residual) 1-alpha (hybrid_pr.cu:43-52).
__global__ void k_pr_init(double *x, double *r, uint32_t nv, double r0) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride) {
    x[v] = 0.0;
    r[v] = r0;
  }
}

// Warm start from a previous solution x0 (kept in x): push values
// pv = alpha * x0 / outdeg and a zeroed residual; after one sweep
// r = sum over in-edges of pv, k_pr_warm_res turns it into the residual of x0,
// r = (1 - alpha) + alpha P^T x0 - x0, so that x0 + (I - alpha P^T)^-1 r is
// the fixed point and the rounds continue from there.
__global__ void k_pr_warm_pv(GraphView g, const double *x, double *pv, double *r, double alpha) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < g.nv; v += stride) {
    const uint32_t l = g.live[v];
    pv[v] = l ? alpha * x[v] / (double)l : 0.0;
    r[v] = 0.0;
  }
}
__global__ void k_pr_warm_res(const double *x, double *r, uint32_t nv, double base) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride)
    r[v] = base + r[v] - x[v];
}

// Absorb of round k: value += w residual, residual = (1 - w) residual (zero in
// a plain round, w = 1), push value w alpha residual / outdeg
// (CombineValueBuffer, hybrid_pr.cu:66-85), so that the sweep makes the
// residual (1 - w) r + w alpha P^T r.  The round's length comes from the
// history (sgs_steplen.cuh), to which the L1 norm of the absorbed residual is
// added; the fit compares it with the previous round's, which the push values
// still hold for the vertices that have out-edges (the others' residuals are
// never passed on).  A snapshot of 10,000 + 10,000 edges at scale 16 and of
// 250,000 + 250,000 on 2 million vertices, result read to the host: 3.35 ->
// 1.61 ms and 28.3 -> 9.6 ms.
// Coherent: r was written earlier in the same launch by other CTAs (the
// persistent round kernel), so it is read through L2.
template <bool Coherent, int N>
__device__ __forceinline__ StepRule pr_absorb_body(const GraphView &g, double *x, double *r, double *pv,
                                                   double alpha, double tol, const StepHist &h, uint32_t k) {
  const StepRule rule = step_rule(h, k, alpha, tol);
  const double w = rule.w;
  const double back = rule.mu / alpha;  // push value * outdeg * back = mu * previous residual
  double acc = 0.0, fit = 0.0;
  // N vertices per thread and step, everything they need requested before
  // anything is used: four where a thread has more than that, one in the
  // launch that runs all rounds, whose graphs have about a vertex per thread, and
  // where the registers of four would halve the CTAs that fit.
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v0 < g.nv; v0 += N * stride) {
    double rv[N], xv[N], prev[N];
    uint32_t l[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint64_t v = v0 + i * stride;
      const bool in = v < g.nv;
      rv[i] = in ? (Coherent ? __ldcg(r + v) : r[v]) : 0.0;
      xv[i] = in ? x[v] : 0.0;
      prev[i] = in && rule.mu > 0.0 ? pv[v] : 0.0;
      l[i] = in ? g.live[v] : 0u;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const uint64_t v = v0 + i * stride;
      if (v >= g.nv) break;
      double p = 0.0;
      if (rv[i] != 0.0) {
        r[v] = w == 1.0 ? 0.0 : (1.0 - w) * rv[i];
        x[v] = xv[i] + w * rv[i];
        acc += fabs(rv[i]);
        if (l[i]) p = w * alpha * rv[i] / (double)l[i];
      }
      if (rule.mu > 0.0 && l[i]) fit += fabs(rv[i] - back * prev[i] * (double)l[i]);
      pv[v] = p;
    }
  }
  __shared__ double s_acc[RELAX_THREADS / 32], s_fit[RELAX_THREADS / 32];
  acc = warp_sum(acc);
  fit = warp_sum(fit);
  if ((threadIdx.x & 31) == 0) {
    s_acc[threadIdx.x >> 5] = acc;
    s_fit[threadIdx.x >> 5] = fit;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0, tf = 0.0;
#pragma unroll
    for (int i = 0; i < RELAX_THREADS / 32; ++i) {
      ta += s_acc[i];
      tf += s_fit[i];
    }
    if (ta != 0.0) atomicAdd(h.l1() + k, ta);
    if (tf != 0.0) atomicAdd(h.fit() + k, tf);
    if (blockIdx.x == 0) record_rule(h, k, rule);
  }
  return rule;
}

template <int N>
__global__ void k_pr_absorb(GraphView g, double *x, double *r, double *pv,
                            double alpha, double tol, StepHist h, uint32_t k) {
  pr_absorb_body<false, N>(g, x, r, pv, alpha, tol, h, k);
}

// PageRank rounds r0, r0+1, ... (at most `limit`) of the pull form in one
// cooperative launch: absorb, grid barrier, pull sweep over the dense
// in-store frontier `fin`, grid barrier, then every thread reads the round's
// absorbed L1 (complete after the barrier) and all stop together once it is
// below the tolerance -- the rounds of the launch-per-kernel loop, in the same
// order, without a launch pair per round and a host read per few rounds
// (which dominate when the graph sits in L2).  *rounds_out = rounds run.
// r and pv are written by other CTAs within the launch and read through L2.
__global__ void __launch_bounds__(RELAX_THREADS)
    k_pr_rounds(GraphView g, FrontierView fin, GraphView gi, double *x, double *r, double *pv,
                double alpha, double tol, StepHist h, uint32_t r0, uint32_t limit,
                unsigned long long *edge_stat, uint32_t *rounds_out) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  uint32_t k = 0;
  while (k < limit) {
    const StepRule rule = pr_absorb_body<true, 1>(g, x, r, pv, alpha, tol, h, r0 + k);
    grid.sync();
    pull_pr_body<true>(fin, gi, pv, r, rule.w != 1.0, edge_stat);
    grid.sync();
    const double l1v = __ldcg(h.l1() + r0 + k);
    ++k;
    if (StepRule::ends(rule.w, l1v, rule.state, tol)) break;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *rounds_out = k;
}

// ---------------------------------------------------------------------------
// Batch apply
// ---------------------------------------------------------------------------
// A batch's inserts and deletes as one list of sort keys, inserts first once
// sorted: delete flag | source | destination in 2 bits + 1 bits (bits =
// those of a vertex id).  One radix sort of both in 2 bits + 1 bits takes 5
// to 7 passes where two sorts of (source << 32 | destination) took 6 or 7
// each; a pass costs about 8 us up to some 10^5 keys, whatever their number.
// Snapshot of 10,000 + 10,000 at scale 16: 934 -> 805 us, with one filter instead
// of a flag pass and two library selections.
__global__ void k_batch_keys(const uint32_t *isrc, const uint32_t *idst, const uint32_t *iw, uint64_t ni,
                             const uint32_t *dsrc, const uint32_t *ddst, uint64_t nd, uint32_t nv, int bits,
                             uint64_t *keys, uint32_t *vals, unsigned int *err) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ni + nd; i += stride) {
    const bool del = i >= ni;
    const uint64_t j = del ? i - ni : i;
    const uint32_t u = (del ? dsrc : isrc)[j], v = (del ? ddst : idst)[j];
    if (u >= nv || v >= nv) atomicOr(err, 1u);
    if (vals) {
      const uint32_t w = del ? 1u : iw[j];
      if (w == 0) atomicOr(err, 2u);
      vals[i] = w;
    }
    keys[i] = ((uint64_t)del << (2 * bits)) | ((uint64_t)u << bits) | v;
  }
}
__device__ __forceinline__ uint64_t edge_of_key(uint64_t k, int bits) {
  const uint64_t mask = (1ull << bits) - 1;
  return ((k >> bits & mask) << 32) | (k & mask);
}

// Deletes of the sorted list as (source << 32 | destination); with `ins` the
// inserts too.
__global__ void k_expand_keys(const uint64_t *keys, uint64_t ni, uint64_t nd, int bits, uint64_t *ins,
                              uint64_t *del) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ni + nd; i += stride) {
    if (i >= ni) del[i - ni] = edge_of_key(keys[i], bits);
    else if (ins) ins[i] = edge_of_key(keys[i], bits);
  }
}

__device__ __forceinline__ bool sorted_has(const uint64_t *a, uint32_t n, uint64_t k) {
  uint32_t l = 0, r = n;
  while (l < r) {
    uint32_t m = (l + r) >> 1;
    if (a[m] < k) l = m + 1;
    else r = m;
  }
  return l < n && a[l] == k;
}

// The inserts that survive the batch's deletes (insert-then-delete order of
// framework.cuh:1011-1012), in order, in two launches of the same grid over
// the same contiguous shares: flags and kept counts per CTA, then every CTA
// adds up the counts before its own and writes its share.  The first also
// expands the deletes.
__global__ void __launch_bounds__(256)
    k_filter_inserts(const uint64_t *keys, uint32_t n_ins, uint32_t n_del, int bits, unsigned char *flag,
                     uint32_t *counts, uint64_t *del_out) {
  const uint64_t *del = keys + n_ins;
  const uint64_t dbit = 1ull << (2 * bits);
  const uint32_t share = (n_ins + gridDim.x - 1) / gridDim.x;
  const uint64_t b = (uint64_t)blockIdx.x * share, e = min(b + share, (uint64_t)n_ins);
  uint32_t kept = 0;
  for (uint64_t i = b + threadIdx.x; i < e; i += blockDim.x) {
    const bool k = !n_del || !sorted_has(del, n_del, keys[i] | dbit);
    flag[i] = k;
    kept += k;
  }
  __shared__ uint32_t s_kept;
  if (threadIdx.x == 0) s_kept = 0;
  __syncthreads();
  kept = warp_sum(kept);
  if ((threadIdx.x & 31) == 0 && kept) atomicAdd(&s_kept, kept);
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = s_kept;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_del; i += stride)
    del_out[i] = edge_of_key(del[i], bits);
}
__global__ void __launch_bounds__(256)
    k_keep_inserts(const uint64_t *keys, const uint32_t *vals, uint32_t n_ins, int bits,
                   const unsigned char *flag, const uint32_t *counts, uint64_t *ins_out, uint32_t *w_out,
                   uint32_t *n_kept) {
  __shared__ uint32_t s_base, s_warp[8];
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_base = 0;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t c = threadIdx.x; c < blockIdx.x; c += blockDim.x) before += counts[c];
  before = warp_sum(before);
  if (lane == 0 && before) atomicAdd(&s_base, before);
  __syncthreads();
  uint32_t at = s_base;
  const uint32_t share = (n_ins + gridDim.x - 1) / gridDim.x;
  const uint64_t b = (uint64_t)blockIdx.x * share, e = min(b + share, (uint64_t)n_ins);
  for (uint64_t t = b; t < e; t += 256) {
    const uint64_t i = t + threadIdx.x;
    const bool keep = i < e && flag[i];
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, keep);
    if (lane == 0) s_warp[wid] = __popc(m);
    __syncthreads();
    uint32_t pos = at, all = 0;
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
      pos += q < wid ? s_warp[q] : 0u;
      all += s_warp[q];
    }
    if (keep) {
      pos += __popc(m & ((1u << lane) - 1u));
      ins_out[pos] = edge_of_key(keys[i], bits);
      if (w_out) w_out[pos] = vals[i];
    }
    at += all;
    __syncthreads();  // s_warp is rewritten by the next step
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *n_kept = at;
}

// One entry per distinct source of a sorted key list (group heads); aux =
// group start.  With `mark`, sources already marked with `stamp` are skipped,
// which builds the union of the sources of several lists.
__global__ void k_group_heads(GraphView g, const uint64_t *keys,
                              const uint32_t *n_ptr, uint32_t n_fixed,
                              uint32_t *gstart, uint32_t *mark, uint32_t stamp,
                              FrontierView out) {
  const uint32_t n = n_ptr ? *n_ptr : n_fixed;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < n; b += stride) {
    const uint64_t i = b + threadIdx.x;
    bool want = false;
    uint32_t u = 0, d = 0;
    if (i < n) {
      u = (uint32_t)(keys[i] >> 32);
      const bool head = i == 0 || (uint32_t)(keys[i - 1] >> 32) != u;
      if (head) {
        d = g.slots[u];
        want = d > 0;
        if (want && mark) want = atomicExch(&mark[u], stamp) != stamp;
      }
    }
    frontier_append_block(out, want, u, d, gstart, (uint32_t)i);
  }
}

// Insert phase 1 (one thread per distinct source of the kept, sorted inserts):
// append in place when the block has room, else relocate the block to a new
// region of the same tier (capacity grows 1.5x) and queue the copy of the old
// slots.  Mirrors PMAGraph::insert's "append at index+degree" and its
// resize-on-overflow, without shifting neighbours.
struct InsertCtx {
  unsigned long long *arena_top;   // [2] per tier
  uint64_t arena_cap[2];
  unsigned int *err;
  uint64_t *wbase;                 // per vertex: write position of its inserts
  // relocation list
  uint32_t *rl_vtx;
  uint64_t *rl_from;
  uint64_t *rl_to;
  uint32_t *rl_len;
  unsigned long long *rl_count64;
  unsigned long long *fit;         // 0: no room, nothing is changed
};

__device__ __forceinline__ uint32_t grow_cap(uint32_t need) {
  uint64_t c = (uint64_t)need + (need >> 1) + 4;
  c = (c + 3) & ~3ull;
  return (uint32_t)min(c, (uint64_t)0xFFFFFFF0u);
}

// Between the dry run and the plan: whether the relocations fit the arenas.
// `again`: they were made to.
__global__ void k_insert_fits(InsertCtx c, const unsigned long long *demand, bool again) {
  *c.fit = again || (c.arena_top[0] + demand[0] <= c.arena_cap[0] && c.arena_top[1] + demand[1] <= c.arena_cap[1]);
}

__global__ void k_insert_plan(GraphView g, const uint64_t *keys, const uint32_t *n_ptr,
                              InsertCtx c, int dry, unsigned long long *demand) {
  if (!dry && !*c.fit) return;
  const uint32_t n = *n_ptr;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < n; b += stride) {
    const uint64_t i = b + threadIdx.x;
    // per-lane decision; the arena/demand/relocation atomics are warp-aggregated
    bool head = false, reloc = false;
    uint32_t u = 0, k = 0, sl = 0, nc = 0;
    uint64_t o = 0;
    int tier = 0;
    if (i < n) {
      u = (uint32_t)(keys[i] >> 32);
      head = i == 0 || (uint32_t)(keys[i - 1] >> 32) != u;
    }
    if (head) {
      // group end: exponential then binary search (groups are usually tiny)
      const uint64_t lim = ((uint64_t)u + 1) << 32;
      uint32_t lo = (uint32_t)i + 1, step = 1, hi = lo;
      while (hi < n && keys[hi] < lim) {
        lo = hi + 1;
        hi = (uint32_t)min((uint64_t)hi + step, (uint64_t)n);
        step <<= 1;
      }
      while (lo < hi) {
        const uint32_t m = (lo + hi) >> 1;
        if (keys[m] < lim) lo = m + 1;
        else hi = m;
      }
      k = lo - (uint32_t)i;
      sl = g.slots[u];
      const uint32_t cp = g.cap[u];
      const uint64_t need = (uint64_t)sl + k;
      o = g.off[u];
      tier = (o & HOST_BIT) ? 1 : 0;
      if (need <= cp) {
        if (!dry) {
          c.wbase[u] = o + sl;
          g.slots[u] = (uint32_t)need;
          g.live[u] += k;
        }
      } else if (need > 0xFFFFFFF0ull) {
        atomicOr(c.err, 4u);
      } else {
        reloc = true;
        nc = grow_cap((uint32_t)need);
      }
    }
    if (dry) {
      for (int t = 0; t < 2; ++t) warp_atomic_add(&demand[t], reloc && tier == t, nc);
      continue;
    }
    unsigned long long pos[2];
    for (int t = 0; t < 2; ++t) pos[t] = warp_atomic_add(&c.arena_top[t], reloc && tier == t, nc);
    const unsigned long long q =
        warp_atomic_add((unsigned long long *)c.rl_count64, reloc && sl > 0, 1ull);
    if (reloc) {
      const unsigned long long p0 = pos[tier];
      if (p0 + nc > c.arena_cap[tier]) {
        atomicOr(c.err, 8u);
      } else {
        const uint64_t no = p0 | (tier ? HOST_BIT : 0);
        if (sl) {
          c.rl_vtx[q] = u;
          c.rl_from[q] = o;
          c.rl_to[q] = no;
          c.rl_len[q] = sl;
        }
        c.wbase[u] = no + sl;
        g.off[u] = no;
        g.cap[u] = nc;
        g.slots[u] = sl + k;
        g.live[u] += k;
      }
    }
  }
}

// Insert phase 2: one thread per kept insert writes (dst, w) at its rank
// within its source's group.
__global__ void k_insert_write(GraphView g, const uint64_t *keys, const uint32_t *w,
                               const uint32_t *n_ptr, InsertCtx c) {
  if (!*c.fit) return;
  const uint64_t *wbase = c.wbase;
  const uint32_t n = *n_ptr;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint64_t k = keys[i];
    const uint32_t u = (uint32_t)(k >> 32), v = (uint32_t)k;
    // group start: exponential search backwards, then binary search
    const uint64_t lo_key = (uint64_t)u << 32;
    uint32_t hi = (uint32_t)i, step = 1, lo = hi;
    while (lo > 0 && keys[lo - 1] >= lo_key) {
      hi = lo - 1;
      lo = lo > step ? lo - step : 0;
      step <<= 1;
    }
    while (lo < hi) {
      const uint32_t m = (lo + hi) >> 1;
      if (keys[m] < lo_key) lo = m + 1;
      else hi = m;
    }
    const uint64_t pos = wbase[u] + (i - lo);
    const bool ew = g.wmode == W_EXPLICIT;
    store_slot(g, pos, 0, v, ew, ew ? w[i] : 0u);
  }
}

// Relocation list -> frontier of copy entries; the entry's vertex field holds
// the relocation list index.
__global__ void k_reloc_frontier(const unsigned long long *rl_count, const uint32_t *rl_len,
                                 FrontierView out) {
  const uint32_t n = (uint32_t)*rl_count;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x; b < n; b += stride) {
    const uint64_t i = b + threadIdx.x;
    const uint32_t d = i < n ? rl_len[i] : 0u;
    frontier_append(out, d > 0, (uint32_t)i, d);
  }
}

// Copy op over relocation entries: vertex field = relocation list index.
// Tombstone reclamation.  The reference's del_edge shifts the rest of the
// list left on every delete (csr_graph.cuh:789-811) and its PMA rebalances
// windows by density (:813-933).  Here a snapshot's deletes only write
// tombstones, and then every block they touched whose dead slots reach a
// sixteenth of its live ones is compacted in place: one warp per block reads 32
// slots at a time, keeps the live ones (ballot + prefix) and writes them
// forward, so the block's used slots become its live count and the next
// inserts append right after them.  Each compaction costs at most 17 times
// the slots it reclaims, and no block walked by a relaxation keeps more than
// a sixteenth of dead slots.  Input: the frontier of the touched blocks (one
// entry per source); reclaimed slots are added to *reclaimed.  A block of
// COMPACT_LARGE slots or more (the hubs, which lose edges in every snapshot
// and cross the threshold together) is not walked by a warp, whose steps
// each wait for one load: its vertex goes to `big` (count in big_n) for
// k_compact_large, a CTA per block.
constexpr uint32_t COMPACT_LARGE = 1024;
__global__ void k_compact_blocks(GraphView g, FrontierView f, unsigned long long *reclaimed,
                                 uint32_t *big, uint32_t *big_n) {
  const uint32_t n = (uint32_t)(__ldcg((const unsigned long long *)f.counter) >> CNT_SHIFT);
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const bool ew = g.wmode == W_EXPLICIT;
  unsigned long long got = 0;
  // A warp looks at up to 32 touched blocks at a time, a lane each (fewer when
  // the list is short, so that all warps get some), then compacts the due ones
  // one after the other, the first slots of the next loaded while it works on
  // one.  A warp per block spent a chain of reads on every block, also on
  // those that stay as they are.
  const uint32_t per = (uint32_t)min((n + nwarps - 1) / nwarps, (uint64_t)32);
  for (uint64_t i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (uint64_t)per; i0 < n; i0 += nwarps * per) {
    uint32_t mv = 0, msl = 0;
    uint64_t mo = 0;
    bool due = false;
    if (lane < per && i0 + lane < n) {
      mv = __ldcg(&f.vtx[i0 + lane]);
      msl = g.slots[mv];
      const uint32_t lv = g.live[mv], dead = msl - lv;
      due = dead != 0 && (uint64_t)dead * 16 >= lv;
      if (due && msl >= COMPACT_LARGE) {
        big[atomicAdd(big_n, 1u)] = mv;
        due = false;
      }
      if (due) mo = g.off[mv];
    }
    struct Step {
      uint32_t id, w;
    };
    auto load = [&](uint64_t o, uint32_t j, uint32_t sl) {
      const uint32_t k = j + lane;
      return Step{k < sl ? __ldcg(adj_wptr(g, o) + k) : SGS_TOMB,
                  (ew && k < sl) ? __ldcg(wgt_wptr(g, o) + k) : 0u};
    };
    uint32_t todo = __ballot_sync(0xFFFFFFFFu, due);
    uint64_t o = 0;
    uint32_t sl = 0;
    Step st{SGS_TOMB, 0};
    if (todo) {
      const int from = __ffs(todo) - 1;
      o = __shfl_sync(0xFFFFFFFFu, mo, from);
      sl = __shfl_sync(0xFFFFFFFFu, msl, from);
      st = load(o, 0, sl);
    }
    while (todo) {
      const int from = __ffs(todo) - 1;
      todo &= todo - 1;
      uint64_t no = 0;
      uint32_t nsl = 0;
      Step nst{SGS_TOMB, 0};
      if (todo) {
        const int nf = __ffs(todo) - 1;
        no = __shfl_sync(0xFFFFFFFFu, mo, nf);
        nsl = __shfl_sync(0xFFFFFFFFu, msl, nf);
        nst = load(no, 0, nsl);
      }
      uint32_t out = 0;
      for (uint32_t j = 0; j < sl; j += 32) {
        // every lane's reads of this step and the next are done before any
        // write; writes land at or below the positions of this step
        const Step nx = load(o, j + 32, sl);
        const bool keep = st.id != SGS_TOMB;
        const uint32_t b = __ballot_sync(0xFFFFFFFFu, keep);
        __syncwarp();
        const uint32_t to = out + __popc(b & ((1u << lane) - 1u));
        if (keep && to != j + lane) store_slot(g, o, to, st.id, ew, st.w);  // (not those that stay)
        out += __popc(b);
        st = nx;
        __syncwarp();
      }
      if ((int)lane == from) g.slots[mv] = out;
      if (lane == 0) got += sl - out;
      o = no;
      sl = nsl;
      st = nst;
    }
  }
  if (lane == 0 && got) atomicAdd(reclaimed, got);
}

// In-place compaction of the large blocks listed by k_compact_blocks, one
// CTA per block, in tiles of 4 * COMPACT_THREADS slots: every thread loads a
// 16-B quad of ids (and weights), the CTA scans the live counts and writes
// the live slots forward.  A tile's writes land at or below the positions it
// read, all of which were read before the first barrier of the tile, and
// below the next tile's first slot, so the next tile is loaded before the
// current one is written (software pipeline).  Blocks start on a 4-slot
// boundary and hold a multiple of 4 slots of capacity, so a quad read past
// the used slots stays inside the block.
constexpr int COMPACT_THREADS = 512;
__global__ void __launch_bounds__(COMPACT_THREADS)
    k_compact_large(GraphView g, const uint32_t *big, const uint32_t *big_n, unsigned long long *reclaimed) {
  constexpr int NW = COMPACT_THREADS / 32;
  constexpr uint32_t TILE = 4u * COMPACT_THREADS;
  __shared__ uint32_t s_warp[NW];
  __shared__ uint32_t s_tot;
  const uint32_t n = __ldcg(big_n);
  const bool ew = g.wmode == W_EXPLICIT;
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const uint4 none = make_uint4(SGS_TOMB, SGS_TOMB, SGS_TOMB, SGS_TOMB);
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint32_t v = __ldcg(&big[i]);
    const uint32_t sl = g.slots[v];
    const uint64_t o = g.off[v];
    const uint32_t *a = adj_wptr(g, o);
    const uint32_t *wt = ew ? wgt_wptr(g, o) : nullptr;
    auto load = [&](uint32_t j, uint4 &ids, uint4 &ws) {
      const uint32_t k0 = j + 4 * threadIdx.x;
      ids = none;
      ws = make_uint4(0, 0, 0, 0);
      if (k0 < sl) {
        ids = __ldcg(reinterpret_cast<const uint4 *>(a + k0));
        if (ew) ws = __ldcg(reinterpret_cast<const uint4 *>(wt + k0));
      }
    };
    uint4 ids, ws;
    load(0, ids, ws);
    uint32_t out = 0;  // CTA-uniform
    for (uint32_t j = 0; j < sl; j += TILE) {
      uint4 nids = none, nws = make_uint4(0, 0, 0, 0);
      if (j + TILE < sl) load(j + TILE, nids, nws);
      const uint32_t k0 = j + 4 * threadIdx.x;
      uint32_t keep = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k0 + k < sl && quad_at(ids, k) != SGS_TOMB) keep |= 1u << k;
      const uint32_t c = __popc(keep);
      uint32_t x = c;  // inclusive scan over the warp
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if (lane >= (uint32_t)d) x += y;
      }
      if (lane == 31) s_warp[wid] = x;
      __syncthreads();
      if (wid == 0) {
        const uint32_t t = lane < (uint32_t)NW ? s_warp[lane] : 0u;
        uint32_t u = t;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, u, d);
          if (lane >= (uint32_t)d) u += y;
        }
        if (lane < (uint32_t)NW) s_warp[lane] = u - t;
        if (lane == NW - 1) s_tot = u;
      }
      __syncthreads();
      uint32_t pos = out + s_warp[wid] + x - c;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (keep >> k & 1u) {
          if (pos != k0 + k) store_slot(g, o, pos, quad_at(ids, k), ew, quad_at(ws, k));
          ++pos;
        }
      out += s_tot;
      __syncthreads();  // s_warp / s_tot are rewritten by the next tile
      ids = nids;
      ws = nws;
    }
    if (threadIdx.x == 0) {
      g.slots[v] = out;
      if (sl > out) atomicAdd(reclaimed, (unsigned long long)(sl - out));
    }
  }
}

struct RelocCopyOp {
  static constexpr bool kAppends = false;
  static constexpr bool kQuad = false;
  using Payload = CopyPay;
  GraphView g;
  const uint64_t *rl_from;
  const uint64_t *rl_to;
  __device__ __forceinline__ Payload load(uint32_t, uint32_t q) const {
    CopyPay p;
    p.from = rl_from[q];
    p.to = rl_to[q];
    return p;
  }
  __device__ __forceinline__ uint32_t visit(uint32_t, const Payload &p, uint32_t j,
                                            bool &, uint32_t &, uint32_t &) const {
    const bool ew = g.wmode == W_EXPLICIT;
    store_slot(g, p.to, j, *adj_at(g, p.from, j), ew, ew ? *wgt_at(g, p.from, j) : 0u);
    return 0;
  }
};

// Per-vertex block layout for a fresh arena: capacity with slack.
__global__ void k_layout_caps(const uint32_t *deg, uint32_t nv, uint32_t slack_div,
                              uint32_t *cap) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride) {
    const uint32_t d = deg[v];
    uint64_t c = d ? (uint64_t)d + (slack_div ? d / slack_div : 0) + 2 : 0;
    c = (c + 3) & ~3ull;
    cap[v] = (uint32_t)min(c, (uint64_t)0xFFFFFFF0u);
  }
}

// Device-side validation of a caller CSR: offsets start at 0 and do not
// decrease, destinations < nv, explicit weights >= 1.
__global__ void k_validate_csr(const uint64_t *row, const uint32_t *col, const uint32_t *w,
                               uint32_t nv, uint64_t ne, unsigned int *err) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid == 0 && row[0] != 0) atomicOr(err, 4u);
  for (uint64_t v = tid; v < nv; v += stride)
    if (row[v + 1] < row[v]) atomicOr(err, 4u);
  for (uint64_t i = tid; i < ne; i += stride) {
    if (col[i] >= nv) atomicOr(err, 1u);
    if (w && w[i] == 0) atomicOr(err, 2u);
  }
}

__global__ void k_row_degrees(const uint64_t *row, uint32_t nv, uint32_t *deg) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride)
    deg[v] = (uint32_t)(row[v + 1] - row[v]);
}

// Assign tiers: vertices [0, split) in HBM, the rest in the host arena; the
// offsets come from an exclusive scan of capacities per tier.
__global__ void k_assign_off(const uint64_t *scan, uint32_t nv, uint32_t split,
                             uint64_t host_base_scan, uint64_t *off) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride)
    off[v] = v < split ? scan[v] : ((scan[v] - host_base_scan) | HOST_BIT);
}

__global__ void k_u32_to_u64(const uint32_t *a, uint32_t n, uint64_t *b) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    b[i] = a[i];
}

// ---------------------------------------------------------------------------
// Device R-MAT generator: bit-identical to the oracle's sgso_rmat_edge.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t fin64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
constexpr uint64_t GAMMA = 0x9E3779B97F4A7C15ull;

__global__ void k_rmat(uint32_t scale, uint64_t ne, uint64_t key, uint64_t tA,
                       uint64_t tAB, uint64_t tABC, int drop_self, uint64_t *keys) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < ne; k += stride) {
    uint32_t uu = 0, vv = 0;
    for (uint32_t l = 0; l < scale; ++l) {
      const uint64_t r = fin64(key + (k * 64u + l + 1) * GAMMA) >> 11;
      uint32_t bu, bv;
      if (r < tA) { bu = 0; bv = 0; }
      else if (r < tAB) { bu = 0; bv = 1; }
      else if (r < tABC) { bu = 1; bv = 0; }
      else { bu = 1; bv = 1; }
      uu = (uu << 1) | bu;
      vv = (vv << 1) | bv;
    }
    keys[k] = (drop_self && uu == vv) ? ~0ull : (((uint64_t)uu << 32) | vv);
  }
}

// Weight of edge (u,v) = 1 + top 6 bits of fin64(wkey ^ (u<<32|v)): uniform in
// [1,64]; identical to the oracle's sgso_weight_of.
__global__ void k_hash_weights(const uint64_t *keys, const uint32_t *n_ptr, uint64_t wkey,
                               uint32_t *w) {
  const uint32_t n = *n_ptr;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    w[i] = 1u + (uint32_t)(fin64(wkey ^ keys[i]) >> 58);
}

// row[v] = first index of a key with source >= v in a sorted key list.
__global__ void k_row_from_sorted(const uint64_t *keys, const uint32_t *n_ptr, uint32_t nv,
                                  uint64_t *row) {
  const uint32_t n = *n_ptr;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= nv; v += stride) {
    const uint64_t k = v << 32;
    uint32_t l = 0, r = n;
    while (l < r) {
      uint32_t m = (l + r) >> 1;
      if (keys[m] < k) l = m + 1;
      else r = m;
    }
    row[v] = l;
  }
}

__global__ void k_keys_low(const uint64_t *keys, const uint32_t *n_ptr, uint32_t *col) {
  const uint32_t n = *n_ptr;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    col[i] = (uint32_t)keys[i];
}

__global__ void k_summary_pr(const double *x, uint32_t nv, double *out) {
  double sum = 0.0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride) sum += x[v];
  typedef cub::BlockReduce<double, RELAX_THREADS> BR;
  __shared__ typename BR::TempStorage tmp;
  const double s = BR(tmp).Sum(sum);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

}  // namespace sgs
