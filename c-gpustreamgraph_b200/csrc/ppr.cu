// ppr.cu -- weighted (personalized) PageRank with a hand-written adjoint.
//
// Fixed point (the reference's unnormalised PageRank of
// samples/hybrid_pr/hybrid_pr.cu:26-151 generalised to edge weights and
// teleport vectors): for each of K teleport vectors t_k,
//     x_k = (1 - alpha) t_k + alpha P^T x_k,   P[u,v] = w_uv / s_u, s_u = sum_v w_uv
// (rows without out-edges drop their mass, as in the reference).  With
// t_k = 1 and unit weights this is exactly the reference's PageRank.
//
// Adjoint for an upstream gradient G = dL/dX:
//     Y = G + alpha P Y                       (transposed fixed point)
//     dL/dT = (1 - alpha) Y
//     dL/dw_uv = (1/s_u) sum_k X[u,k] (alpha Y[v,k] - Y[u,k] + G[u,k])
// (the derivative of the row normalisation included; parallel edges each get
// the same term).  All state is FP64, vertex-major [nv][K], so the K values of
// one vertex are one contiguous row of 8K bytes.
//
// Both fixed points are Jacobi iterations of one gather,
//     out[v,:] = c B[v,:] + alpha sum_{i in adj(v)} p_i x[nbr_i, :]
// over the CSC (forward: in-edges) or the CSR (adjoint: out-edges), with the
// edge probabilities p = P[u,v] precomputed once per weight vector.
//
// Work split: a warp owns a work item.  Vertices of at most `piece` edges come
// a few consecutive ones to an item (Impl::items_per_warp); a heavier vertex
// (R-MAT hubs reach 10^5 in-edges) is cut into pieces of that many edges whose
// partial sums go to a scratch row each and are added up, in piece order, by
// the warp that finishes the vertex's last piece -- so no warp walks more than
// `piece` edges of a vertex and a step's result does not depend on the order of
// its items, nor does a step's length (sgs_steplen.cuh).  Inside a warp, LPE
// lanes cover the columns of one neighbour row (CPL columns per lane) and
// 32/LPE neighbours are gathered at once, four deep, so one neighbour row is
// one coalesced read for any K.
#include <cooperative_groups.h>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "../../include/sgs.h"
#include "sgs_steplen.cuh"

namespace sgs {
void set_last_error(const std::string &msg);
}

namespace {

struct PprFail {
  int code;
  std::string msg;
};

void ck(cudaError_t e, const char *what) {
  if (e == cudaSuccess) return;
  cudaGetLastError();
  throw PprFail{e == cudaErrorMemoryAllocation ? SGS_ERR_OOM : SGS_ERR_CUDA,
                std::string(what) + ": " + cudaGetErrorString(e)};
}
#define PCK(x) ck((x), #x)

template <class T>
struct Buf {
  T *p = nullptr;
  size_t n = 0;
  void ensure(size_t want) {
    want = std::max<size_t>(want, 1);
    if (p && want <= n) return;
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
    PCK(cudaMalloc((void **)&p, want * sizeof(T)));
    n = want;
  }
  ~Buf() {
    if (p) cudaFree(p);
  }
};

constexpr int THREADS = 256;
// Most edges of one vertex a warp walks per item, chosen per graph: 128, and 64
// on graphs small enough that the longest walk, not the sum of all, is a step's
// time (4096 vertices, 65536 edges, K = 8, forward and backward: 2.6 ms with
// 256, 1.6 with 64; 2^20 vertices, K = 64: 144 ms with 256 and 32 light
// vertices per item, 102 with 128 and 8).
constexpr uint32_t PIECE_MAX = 128, PIECE_SMALL = 64;
constexpr uint64_t SMALL_EDGES = 2u << 20;

__device__ __forceinline__ uint32_t warp_id() { return (blockIdx.x * blockDim.x + threadIdx.x) >> 5; }
__device__ __forceinline__ uint32_t num_warps() { return (gridDim.x * blockDim.x) >> 5; }

__global__ void k_validate(const uint64_t *row, const uint32_t *col, uint32_t nv, uint64_t ne,
                           unsigned int *err) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid == 0 && row[0] != 0) atomicOr(err, 2u);
  for (uint64_t v = tid; v < nv; v += stride)
    if (row[v + 1] < row[v]) atomicOr(err, 2u);
  for (uint64_t i = tid; i < ne; i += stride)
    if (col[i] >= nv) atomicOr(err, 1u);
}

__global__ void k_edge_src(const uint64_t *row, uint32_t nv, uint32_t *src) {
  const int lane = threadIdx.x & 31;
  for (uint32_t u = warp_id(); u < nv; u += num_warps())
    for (uint64_t e = row[u] + lane; e < row[u + 1]; e += 32) src[e] = u;
}

__global__ void k_iota(uint32_t *a, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    a[i] = (uint32_t)i;
}

// crow[v] = first position of destination >= v in the sorted destinations.
__global__ void k_csc_rows(const uint32_t *sorted_dst, uint64_t ne, uint32_t nv, uint64_t *crow) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= nv;
       v += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t l = 0, r = ne;
    while (l < r) {
      const uint64_t m = (l + r) >> 1;
      if (sorted_dst[m] < v) l = m + 1;
      else r = m;
    }
    crow[v] = l;
  }
}

__global__ void k_gather_u32(const uint32_t *a, const uint32_t *idx, uint64_t n, uint32_t *b) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    b[i] = a[idx[i]];
}

// cnt[v] = number of pieces of v (0 for a vertex of degree <= PIECE); cnt[nv] = 0.
__global__ void k_piece_count(const uint64_t *ptr, uint32_t nv, uint32_t piece, uint32_t *cnt) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v <= nv;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t d = v < nv ? ptr[v + 1] - ptr[v] : 0;
    cnt[v] = d > piece ? (uint32_t)((d + piece - 1) / piece) : 0u;
  }
}

// pv[poff[v] + j] = v for each piece j of v.
__global__ void k_piece_fill(const uint32_t *poff, uint32_t nv, uint32_t *pv) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv;
       v += (uint64_t)gridDim.x * blockDim.x)
    for (uint32_t p = poff[v]; p < poff[v + 1]; ++p) pv[p] = (uint32_t)v;
}

// inv_s[u] = 1 / sum of u's out-edge weights (0 without out-edges) and, with
// pr, the CSR edge probabilities pr[e] = w[e] inv_s[u] of the light vertices;
// err bit 0: a weight that is not positive and finite.  Heavy rows go by their
// pieces (one warp walked a whole hub's row before: 1.6 ms at 2^20 vertices and
// 16.8 M edges, 0.15 now), whose sums the last one to finish adds up in
// piece order; a light row takes 8 lanes, four rows per warp.
__global__ void __launch_bounds__(THREADS)
    k_row_sums(const uint64_t *row, uint32_t nv, const double *w, const uint32_t *pv, const uint32_t *poff,
               uint32_t npieces, uint32_t piece, double *part, uint32_t *done, double *inv_s, double *pr,
               unsigned int *err) {
  constexpr unsigned full = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  bool bad = false;
  for (uint32_t i = warp_id(); i < npieces; i += num_warps()) {
    const uint32_t u = pv[i], first = poff[u], n = poff[u + 1] - first;
    const uint64_t b = row[u] + (uint64_t)(i - first) * piece, e = min(b + piece, row[u + 1]);
    double s = 0.0;
#pragma unroll
    for (uint32_t k = 0; k < PIECE_MAX; k += 32)
      if (b + k + lane < e) {
        const double x = w[b + k + lane];
        bad |= !(x > 0.0) || !isfinite(x);
        s += x;
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(full, s, o);
    uint32_t c = 0;
    if (lane == 0) {
      part[i] = s;
      __threadfence();
      c = atomicAdd(done + first, 1u);
    }
    if (__shfl_sync(full, c, 0) + 1 != n) continue;
    __threadfence();
    double t = 0.0;
    for (uint32_t q = lane; q < n; q += 32) t += __ldcg(part + first + q);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(full, t, o);
    if (lane == 0) {
      done[first] = 0;
      inv_s[u] = t > 0.0 ? 1.0 / t : 0.0;
    }
  }
  const int sub = lane & 7;
  for (uint64_t v0 = (uint64_t)warp_id() * 4; v0 < nv; v0 += (uint64_t)num_warps() * 4) {
    const uint64_t u = v0 + (lane >> 3);
    uint64_t b = 0, e = 0;
    if (u < nv) {
      b = row[u];
      e = row[u + 1];
    }
    const bool light = e - b <= piece;
    if (!light) e = b;
    double s = 0.0;
    for (uint64_t i = b + sub; i < e; i += 8) {
      const double x = w[i];
      bad |= !(x > 0.0) || !isfinite(x);
      s += x;
    }
    __syncwarp();
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(full, s, o);
    const double is = s > 0.0 ? 1.0 / s : 0.0;
    if (u < nv && light && sub == 0) inv_s[u] = is;
    if (pr)
      for (uint64_t i = b + sub; i < e; i += 8) pr[i] = w[i] * is;
  }
  if (bad) atomicOr(err, 1u);
}

// CSR probabilities of the heavy vertices, a warp per piece.
__global__ void k_piece_probs(const uint64_t *row, const double *w, const uint32_t *pv, const uint32_t *poff,
                              uint32_t npieces, uint32_t piece, const double *inv_s, double *pr) {
  const int lane = threadIdx.x & 31;
  for (uint32_t i = warp_id(); i < npieces; i += num_warps()) {
    const uint32_t u = pv[i];
    const uint64_t b = row[u] + (uint64_t)(i - poff[u]) * piece, e = min(b + piece, row[u + 1]);
    const double is = inv_s[u];
    for (uint64_t k = b + lane; k < e; k += 32) pr[k] = w[k] * is;
  }
}

// CSC probabilities: pc[i] = w inv_s of the edge at CSC position i.
__global__ void k_csc_probs(const double *w, const double *inv_s, const uint32_t *ceid, const uint32_t *csrc,
                            uint64_t ne, double *pc) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne;
       i += (uint64_t)gridDim.x * blockDim.x)
    pc[i] = w[ceid[i]] * inv_s[csrc[i]];
}

// Row values: read-only cached loads, or, in the launch that runs many steps
// (it wrote the rows itself, from other SMs too), loads through L2.
template <bool Coh>
__device__ __forceinline__ double ld_row(const double *p) {
  return Coh ? __ldcg(p) : __ldg(p);
}

// Narrow rows (K <= 16): a group of LPE lanes sums the rows of [b, e), LPE lanes
// covering a row's columns and taking every `stride`-th edge, DEPTH at a time.
template <int LPE, int DEPTH, bool Coh>
__device__ __forceinline__ double gather_narrow(const uint32_t *__restrict__ nbr, const double *__restrict__ p,
                                                uint64_t b, uint64_t e, uint32_t stride, uint32_t k, uint32_t K,
                                                const double *x) {
  double acc = 0.0;
  uint64_t i = b;
  for (; i < e; i += DEPTH * stride) {
    uint32_t u[DEPTH];
    double pp[DEPTH], xv[DEPTH];
#pragma unroll
    for (int q = 0; q < DEPTH; ++q) {
      const bool ok = i + q * stride < e;
      u[q] = ok ? __ldg(nbr + i + q * stride) : 0u;
      pp[q] = ok ? __ldg(p + i + q * stride) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < DEPTH; ++q)
      xv[q] = k < K && i + q * stride < e ? ld_row<Coh>(x + (uint64_t)u[q] * K + k) : 0.0;
#pragma unroll
    for (int q = 0; q < DEPTH; ++q) acc = fma(pp[q], xv[q], acc);
  }
  return acc;
}

// Wide rows (K > 16): the warp covers the row's columns kb, kb + 32, ... (CPL
// per lane); acc[j] += sum over [b, e) of p x.  Neighbour ids and
// probabilities come 32 at a time in one coalesced load (the first 32 are
// given: they were loaded ahead) and are handed out by shuffles, so the only
// dependent load per neighbour is its row; DEPTH rows are in flight.
struct Head {
  uint32_t u;
  double p;
};
__device__ __forceinline__ Head load_head(const uint32_t *__restrict__ nbr, const double *__restrict__ p,
                                          uint64_t b, uint64_t e, int lane) {
  return b + lane < e ? Head{__ldg(nbr + b + lane), __ldg(p + b + lane)} : Head{0u, 0.0};
}
template <int CPL, bool Coh>
__device__ __forceinline__ void gather_wide(const uint32_t *__restrict__ nbr, const double *__restrict__ p,
                                            uint64_t b, uint64_t e, Head h, int lane, uint32_t kb, uint32_t K,
                                            const double *x, double (&acc)[CPL]) {
  constexpr int DEPTH = 4;
  for (uint64_t c = b; c < e; c += 32) {
    const uint32_t cnt = e - c < 32 ? (uint32_t)(e - c) : 32u;
    const Head nx = load_head(nbr, p, c + 32, e, lane);
    for (uint32_t r = 0; r < cnt; r += DEPTH) {
      uint32_t u[DEPTH];
      double pp[DEPTH], xv[DEPTH][CPL];
#pragma unroll
      for (int q = 0; q < DEPTH; ++q) {
        u[q] = __shfl_sync(0xFFFFFFFFu, h.u, (r + q) & 31);
        pp[q] = __shfl_sync(0xFFFFFFFFu, h.p, (r + q) & 31);
      }
#pragma unroll
      for (int q = 0; q < DEPTH; ++q)
#pragma unroll
        for (int j = 0; j < CPL; ++j) {
          const uint32_t k = kb + 32 * j;
          xv[q][j] = r + q < cnt && k < K ? ld_row<Coh>(x + (uint64_t)u[q] * K + k) : 0.0;
        }
#pragma unroll
      for (int q = 0; q < DEPTH; ++q)
#pragma unroll
        for (int j = 0; j < CPL; ++j) acc[j] = fma(pp[q], xv[q][j], acc[j]);
    }
    h = nx;
  }
}

// One step's arguments: the edge lists with their pieces, out = x + w d with
// d = c B + alpha sum p x - x, and the history of the step lengths.
struct StepArgs {
  const uint64_t *ptr;
  const uint32_t *nbr;
  const double *p;
  uint32_t nv;
  const uint32_t *pv, *poff;
  uint32_t npieces, piece;
  uint32_t K;
  double alpha, c;
  const double *B;
  double *part;    // a row of K per piece
  uint32_t *done;  // finished pieces, at the vertex's first piece (zero between steps)
  uint32_t *next;  // next item, one counter per step of the history (zero before it)
  uint32_t per;    // light vertices per item
  sgs::StepHist h;
  double tol;
};

// The new state of one entry; |d|, so that the order of the additions does not
// show, and the fit (sgs_steplen.cuh) into dsum, fsum.  out still holds the state before x, so x - out is the previous d.
template <bool Coh>
__device__ __forceinline__ void finish_entry(const StepArgs &a, const sgs::StepRule &rule, uint64_t o, double sum,
                                             const double *x, double *out, double &dsum, double &fsum) {
  const double nx = a.c * __ldg(a.B + o) + a.alpha * sum;
  const double xo = ld_row<Coh>(x + o);
  const double d = nx - xo;
  dsum += sgs::exact_term(fabs(d), rule.unit);
  if (rule.mu > 0.0) fsum += fabs(d - rule.mu * (xo - __ldcg(out + o)));
  out[o] = rule.w == 1.0 ? nx : fma(rule.w, d, xo);
}

// One step over the work items [0, npieces) (pieces of heavy vertices: partial
// sums to part[piece][K]; the warp that finishes a vertex's last piece adds
// them up in piece order and writes the vertex) and then `per` consecutive
// vertices each, of which it handles the light ones.  The pieces come first, so
// their sums are added while the other warps walk the light vertices; a kernel
// of its own for them cost 5 us per step on a small graph and 85 us at a
// million vertices and K = 64.
// Dyn: warps take items from a counter, the next one requested while one is
// handled.  (Degrees follow the ids' bits on R-MAT graphs, and with a fixed
// stride the resident warps averaged 30 % where 50 % were launched.)  The
// looping launch, whose steps are too short for a round trip per item, strides.
// Vertices without edges keep their first value, c B, for good: only step 0
// writes them.  (2^20 vertices, 16.8 M edges, K = 64: 2.46 ms a step with a
// fixed stride, 32 vertices an item and pieces of 256; 1.01 ms now, 10.3 TB/s
// by the bytes of step_bytes, most rows coming from L2.)
template <int LPE, int CPL, bool Coh>
__device__ __forceinline__ void ppr_step_body(const StepArgs &a, const sgs::StepRule &rule, const double *x,
                                              double *out, uint32_t k_hist, bool first_step) {
  constexpr bool Dyn = !Coh;
  constexpr unsigned full = 0xFFFFFFFFu;
  constexpr int NEG = 32 / LPE;
  constexpr int DEEP = Coh || LPE >= 8 ? 8 : 4, GROUP_DEEP = Coh ? 8 : 4;  // loads in flight per lane group
  const int lane = threadIdx.x & 31;
  const int sub = lane % LPE, eg = lane / LPE;
  const uint32_t K = a.K;
  double dsum = 0.0, fsum = 0.0;
  const uint32_t items = a.npieces + (a.nv + a.per - 1) / a.per;
  const uint32_t W = num_warps();
  // the row sums of [b, e) for the whole warp, columns k0 on: every lane ends up
  // with those of its columns (narrow forms: each lane group with all)
  auto row_sums = [&](uint64_t b, uint64_t e, const Head &h, uint32_t k0, double (&acc)[CPL]) {
#pragma unroll
    for (int j = 0; j < CPL; ++j) acc[j] = 0.0;
    if constexpr (LPE == 32) {
      gather_wide<CPL, Coh>(a.nbr, a.p, b, e, h, lane, k0 + lane, K, x, acc);
    } else {
      acc[0] = gather_narrow<LPE, DEEP, Coh>(a.nbr, a.p, b + eg, e, NEG, k0 + sub, K, x);
#pragma unroll
      for (int o = 16; o >= LPE; o >>= 1) acc[0] += __shfl_xor_sync(full, acc[0], o);
    }
  };
  uint32_t it = warp_id();
  if constexpr (Dyn) {
    if (lane == 0) it = atomicAdd(a.next + k_hist, 1u);
    it = __shfl_sync(full, it, 0);
  }
  while (it < items) {
    uint32_t nxt = it + W;
    if constexpr (Dyn) {
      if (lane == 0) nxt = atomicAdd(a.next + k_hist, 1u);
    }
    if (it < a.npieces) {
      const uint32_t v = a.pv[it], first = a.poff[v], last = a.poff[v + 1];
      const uint64_t b = a.ptr[v] + (uint64_t)(it - first) * a.piece, e = min(b + a.piece, a.ptr[v + 1]);
      const Head h = LPE == 32 ? load_head(a.nbr, a.p, b, e, lane) : Head{0u, 0.0};
      for (uint32_t k0 = 0; k0 < K; k0 += LPE * CPL) {
        double acc[CPL];
        row_sums(b, e, h, k0, acc);
        if (eg == 0) {
#pragma unroll
          for (int j = 0; j < CPL; ++j) {
            const uint32_t k = k0 + sub + j * LPE;
            if (k < K) a.part[(uint64_t)it * K + k] = acc[j];
          }
        }
      }
      __threadfence();  // this warp's row before its count
      __syncwarp();
      uint32_t n = 0;
      if (lane == 0) n = atomicAdd(a.done + first, 1u);
      n = __shfl_sync(full, n, 0);
      if (n + 1 == last - first) {
        __threadfence();
        if (lane == 0) a.done[first] = 0;
        for (uint32_t k = lane; k < K; k += 32) {
          double sum = 0.0;
#pragma unroll 8
          for (uint32_t q = first; q < last; ++q) sum += __ldcg(a.part + (uint64_t)q * K + k);
          finish_entry<Coh>(a, rule, (uint64_t)v * K + k, sum, x, out, dsum, fsum);
        }
      }
    } else {
      const uint32_t v0 = (it - a.npieces) * a.per;
      const uint32_t n = min(a.per, a.nv - v0);
      const uint64_t rb = (uint32_t)lane < n ? a.ptr[v0 + lane] : 0;
      const uint64_t re = (uint32_t)lane < n ? a.ptr[v0 + lane + 1] : 0;
      const uint64_t deg = re - rb;
      if (first_step) {
        for (uint32_t em = __ballot_sync(full, (uint32_t)lane < n && deg == 0); em; em &= em - 1) {
          const uint64_t o = (uint64_t)(v0 + __ffs(em) - 1) * K;
          for (uint32_t k = lane; k < K; k += 32) finish_entry<Coh>(a, rule, o + k, 0.0, x, out, dsum, fsum);
        }
      }
      uint32_t todo = __ballot_sync(full, deg > 0 && deg <= a.piece);
      if constexpr (LPE < 32) {
        // up to 32 edges: a lane group per vertex, NEG vertices at a time;
        uint32_t lo = __ballot_sync(full, deg > 0 && deg <= 32);
        todo &= ~lo;
        // so with heavier ones if that takes fewer loads in a row than the warp on
        // one after the other (20,000 vertices, a fifth of them with 64 in-edges,
        // K = 1: 36 -> 19 us a step)
        const uint32_t many = __popc(todo);
        if ((many + NEG - 1) / NEG * ((a.piece + GROUP_DEEP - 1) / GROUP_DEEP) <
            many * ((a.piece + NEG * DEEP - 1) / (NEG * DEEP))) {
          lo |= todo;
          todo = 0;
        }
        while (lo) {
          const int my = eg < __popc(lo) ? (int)__fns(lo, 0, eg + 1) : -1;
          const uint64_t b = __shfl_sync(full, rb, my & 31), e = __shfl_sync(full, re, my & 31);
          if (my >= 0) {
            const double s = gather_narrow<LPE, GROUP_DEEP, Coh>(a.nbr, a.p, b, e, 1, sub, K, x);
            if ((uint32_t)sub < K) finish_entry<Coh>(a, rule, (uint64_t)(v0 + my) * K + sub, s, x, out, dsum, fsum);
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < NEG; ++q) lo &= lo - 1;
        }
      }
      // one vertex at a time, the next one's first ids and probabilities ahead
      Head h{0u, 0.0};
      uint64_t b = 0, e = 0;
      if (todo) {
        const int f = __ffs(todo) - 1;
        b = __shfl_sync(full, rb, f);
        e = __shfl_sync(full, re, f);
        if constexpr (LPE == 32) h = load_head(a.nbr, a.p, b, e, lane);
      }
      while (todo) {
        const uint32_t v = v0 + __ffs(todo) - 1;
        todo &= todo - 1;
        uint64_t nb = 0, ne = 0;
        Head nh{0u, 0.0};
        if (todo) {
          const int f = __ffs(todo) - 1;
          nb = __shfl_sync(full, rb, f);
          ne = __shfl_sync(full, re, f);
          if constexpr (LPE == 32) nh = load_head(a.nbr, a.p, nb, ne, lane);
        }
        for (uint32_t k0 = 0; k0 < K; k0 += LPE * CPL) {
          double acc[CPL];
          row_sums(b, e, h, k0, acc);
          if (eg == 0) {
#pragma unroll
            for (int j = 0; j < CPL; ++j) {
              const uint32_t k = k0 + sub + j * LPE;
              if (k < K) finish_entry<Coh>(a, rule, (uint64_t)v * K + k, acc[j], x, out, dsum, fsum);
            }
          }
        }
        b = nb;
        e = ne;
        h = nh;
      }
    }
    it = Dyn ? __shfl_sync(full, nxt, 0) : nxt;
  }
  // one atomic per CTA (one per warp, all on one address, cost a small graph's
  // step more than its sums)
  __shared__ double s_d[THREADS / 32], s_f[THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    dsum += __shfl_xor_sync(full, dsum, o);
    fsum += __shfl_xor_sync(full, fsum, o);
  }
  if (lane == 0) {
    s_d[threadIdx.x >> 5] = dsum;
    s_f[threadIdx.x >> 5] = fsum;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double d = 0.0, f = 0.0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
      d += s_d[w];
      f += s_f[w];
    }
    if (d != 0.0) atomicAdd(a.h.l1() + k_hist, d);
    if (f != 0.0) atomicAdd(a.h.fit() + k_hist, f);
    if (blockIdx.x == 0) sgs::record_rule(a.h, k_hist, rule);
  }
}

// (From 5 columns on with 64 registers, and gathers 8 deep up to 16: 2^16 vertices,
// K = 8, 1.00 ms, 1.11 with 48 and 4 deep.)
template <int LPE, int CPL>
__global__ void __launch_bounds__(THREADS, LPE >= 8 ? 4 : 5)
    k_ppr_step(StepArgs a, const double *__restrict__ x, double *out, uint32_t k, bool first) {
  ppr_step_body<LPE, CPL, false>(a, sgs::step_rule<true>(a.h, k, a.alpha, a.tol * sgs::LONG_TOL), x, out, k, first);
}

// The end of the iteration, the same on both sides: a plain step below the
// tolerance that is also a sixteenth of it (LONG_TOL; a second one after a long
// step, sgs_steplen.cuh), or the EXTRA-th one below it, should rounding keep
// the rest away.
// Rounding: the steps' changes no longer fall (`prev`: the change of the step
// before, 0 if that was a long one).
constexpr uint32_t EXTRA = 20;
__host__ __device__ inline bool ppr_ends(double w, double l1, double prev, int state, double tol, double alpha,
                                         uint32_t &under) {
  if (w != 1.0 || !(l1 < tol)) return false;
  ++under;
  return sgs::StepRule::ends(w, l1, state, tol * sgs::LONG_TOL) || under > EXTRA ||
         (prev > 0.0 && l1 > (alpha > 0.9 ? alpha : 0.9) * prev);
}

// Steps k0 .. k1 - 1 in one cooperative launch, a grid barrier after each, until
// the end; step k reads buffer k % 2 and writes the other.  For graphs whose
// step takes about as long as a launch: forward and backward on 4,096 vertices
// with K = 8 took 8.0 ms with two launches per step and 0.84 per step, 2.3 with
// this loop and the long steps.
template <int LPE, int CPL, bool One>
__global__ void __launch_bounds__(THREADS, 4)
    k_ppr_steps(StepArgs a, double *x0, double *x1, uint32_t k0, uint32_t k1, uint32_t under, bool first,
                uint32_t *ran) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  // One: one thread of the CTA reads the history, a step's end and the next one's
  // rule at once.
  __shared__ sgs::StepRule s_rule;
  __shared__ bool s_end;
  auto rule_of = [&](uint32_t k) { return sgs::step_rule<true>(a.h, k, a.alpha, a.tol * sgs::LONG_TOL); };
  auto ends = [&](const sgs::StepRule &rule, uint32_t k) {
    const double norm = __ldcg(a.h.l1() + k), norm1 = __ldcg(a.h.l1() + (k ? k - 1 : 0));
    const double w1 = __ldcg(a.h.step() + (k ? k - 1 : 0));
    return ppr_ends(rule.w, norm + sgs::exact_slack(rule.unit, (double)a.nv * a.K), k && w1 == 1.0 ? norm1 : 0.0,
                    rule.state, a.tol, a.alpha, under);
  };
  uint32_t k = k0;
  if constexpr (One) {
    if (threadIdx.x == 0) s_rule = rule_of(k);
    __syncthreads();
    while (k < k1) {
      ppr_step_body<LPE, CPL, true>(a, s_rule, k % 2 ? x1 : x0, k % 2 ? x0 : x1, k, first && k == k0);
      grid.sync();
      if (threadIdx.x == 0) {
        const sgs::StepRule done = s_rule;
        s_rule = rule_of(k + 1);
        s_end = ends(done, k);
      }
      __syncthreads();
      ++k;
      if (s_end) break;
    }
  } else {
    while (k < k1) {
      const sgs::StepRule rule = rule_of(k);
      ppr_step_body<LPE, CPL, true>(a, rule, k % 2 ? x1 : x0, k % 2 ? x0 : x1, k, first && k == k0);
      grid.sync();
      if (ends(rule, k++)) break;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *ran = k - k0;
}

// gw[e] = inv_s[u] (alpha sum_k X[u,k] Y[v,k] + c_u) for e = (u,v), where
// c_u = sum_k X[u,k] (G[u,k] - Y[u,k]); work items as in k_ppr_step over the
// CSR, taken from a counter.  Bound by the gather of Y's rows: four are in
// flight per lane group, and their dot products are reduced together, halving
// the values held with the lanes they cover (6 exchanges for four sums instead of
// 20).  (2^20 vertices, K = 64: 7.2 ms with fixed strides and a reduction per
// edge, 1.96 now.)
// CPL columns per lane (its X entries stay in registers), LPE lanes per row.
template <int LPE, int CPL>
__global__ void __launch_bounds__(THREADS)
    k_ppr_edge_grad(const uint64_t *__restrict__ row, const uint32_t *__restrict__ col,
                    const double *__restrict__ inv_s, uint32_t nv, const uint32_t *__restrict__ pv,
                    const uint32_t *__restrict__ poff, uint32_t npieces, uint32_t piece, uint32_t K,
                    double alpha, const double *__restrict__ X, const double *__restrict__ Y,
                    const double *__restrict__ G, double *__restrict__ gw, uint32_t *next) {
  constexpr int NEG = 32 / LPE;
  constexpr unsigned full = 0xFFFFFFFFu;
  constexpr uint32_t PER = 8;  // vertices per item
  const int lane = threadIdx.x & 31;
  const int sub = lane % LPE, eg = lane / LPE;
  const uint32_t items = npieces + (nv + PER - 1) / PER;
  auto edges = [&](uint32_t u, uint64_t b, uint64_t e) {
    const uint64_t ou = (uint64_t)u * K;
    const double is = inv_s[u];
    double xu[CPL], cu = 0.0;
    for (uint32_t k = lane; k < K; k += 32) cu += X[ou + k] * (G[ou + k] - Y[ou + k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cu += __shfl_xor_sync(full, cu, o);
#pragma unroll
    for (int j = 0; j < CPL; ++j) xu[j] = sub + j * LPE < K ? X[ou + sub + j * LPE] : 0.0;
    for (uint64_t e0 = b; e0 < e; e0 += 4 * NEG) {
      double t[4];
      uint32_t v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint64_t i = e0 + q * NEG + eg;
        v[q] = i < e ? __ldg(col + i) : 0u;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        t[q] = 0.0;
        const bool ok = e0 + q * NEG + eg < e;
#pragma unroll
        for (int j = 0; j < CPL; ++j)
          if (ok && sub + j * LPE < K) t[q] = fma(xu[j], __ldg(Y + (uint64_t)v[q] * K + sub + j * LPE), t[q]);
        if constexpr (CPL == 2)  // more than 64 columns: the rest of the row
          if (ok)
            for (uint32_t k = sub + CPL * LPE; k < K; k += LPE)
              t[q] = fma(X[ou + k], __ldg(Y + (uint64_t)v[q] * K + k), t[q]);
      }
      if constexpr (LPE >= 4) {
        // four sums over LPE lanes: after two halving steps lane group s / (LPE/4)
        // holds edge q = s / (LPE/4)'s
        const bool up = sub & (LPE / 2);
        double a0 = up ? t[2] : t[0], a1 = up ? t[3] : t[1];
        a0 += __shfl_xor_sync(full, up ? t[0] : t[2], LPE / 2);
        a1 += __shfl_xor_sync(full, up ? t[1] : t[3], LPE / 2);
        const bool up2 = sub & (LPE / 4);
        double z = up2 ? a1 : a0;
        z += __shfl_xor_sync(full, up2 ? a0 : a1, LPE / 4);
#pragma unroll
        for (int o = LPE / 8; o > 0; o >>= 1) z += __shfl_xor_sync(full, z, o);
        const int q = (up ? 2 : 0) + (up2 ? 1 : 0);
        const uint64_t i = e0 + q * NEG + eg;
        if (i < e && sub % (LPE / 4) == 0) gw[i] = is * fma(alpha, z, cu);
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
          for (int o = LPE / 2; o > 0; o >>= 1) t[q] += __shfl_xor_sync(full, t[q], o);
          const uint64_t i = e0 + q * NEG + eg;
          if (i < e && sub == 0) gw[i] = is * fma(alpha, t[q], cu);
        }
      }
    }
  };
  for (;;) {
    uint32_t it = 0;
    if (lane == 0) it = atomicAdd(next, 1u);
    it = __shfl_sync(full, it, 0);
    if (it >= items) break;
    if (it < npieces) {
      const uint32_t u = pv[it];
      const uint64_t b = row[u] + (uint64_t)(it - poff[u]) * piece;
      edges(u, b, min(b + piece, row[u + 1]));
    } else {
      const uint32_t v0 = (it - npieces) * PER;
      for (uint32_t u = v0; u < min(v0 + PER, nv); ++u) {
        const uint64_t b = row[u], e = row[u + 1];
        if (e != b && e - b <= piece) edges(u, b, e);
      }
    }
  }
}

__global__ void k_scale(const double *a, double s, uint64_t n, double *b) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    b[i] = s * a[i];
}

int lanes_per_edge(uint32_t K) {
  int l = 1;
  while (l < 32 && (uint32_t)l < K) l <<= 1;
  return l;
}

// The edge lists of one direction with their heavy-vertex pieces.
struct Adj {
  const uint64_t *ptr = nullptr;
  const uint32_t *nbr = nullptr;
  Buf<uint32_t> poff, pv;
  uint32_t npieces = 0;
};

}  // namespace

// A graph prepared for PPR: the CSR (out-edges) and a CSC (in-edges) whose
// entries carry the CSR index of the edge, so weights given in CSR order
// apply to both directions.
struct sgs_ppr {
  int dev = 0;
  int nsm = 148;
  cudaStream_t s = nullptr;
  uint32_t nv = 0;
  uint64_t ne = 0;
  Buf<uint64_t> row, crow;
  Buf<uint32_t> col, csrc, ceid;
  Buf<double> w, inv_s, pr, pc, t, x, xn, g, y, yn, part;
  // one allocation: the step history, then (u32) the steps' item counters, the
  // steps a looping launch ran and the finished pieces per heavy vertex
  Buf<double> work;
  uint32_t *next() { return (uint32_t *)(work.p + sgs::StepHist::FIELDS * (size_t)HIST); }
  uint32_t *ran() { return next() + HIST; }
  uint32_t *done() { return ran() + 1; }
  static constexpr uint32_t HIST = 512;  // steps the history holds
  Buf<unsigned int> err;
  uint32_t piece = PIECE_MAX;
  Adj in, out;  // CSC (forward) and CSR (adjoint, edge gradient)
  // timing and counters
  bool timing = false;
  std::vector<cudaEvent_t> ev;  // around a batch of steps (timing on)
  cudaEvent_t call_ev[2] = {nullptr, nullptr};
  sgs_ppr_stats st{};
  uint64_t n_launch = 0;
  ~sgs_ppr() {
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
    for (cudaEvent_t e : call_ev)
      if (e) cudaEventDestroy(e);
    if (s) cudaStreamDestroy(s);
  }
  void events() {
    if (!call_ev[0]) {
      PCK(cudaEventCreate(&call_ev[0]));
      PCK(cudaEventCreate(&call_ev[1]));
    }
    while (ev.size() < 2) {
      cudaEvent_t e;
      PCK(cudaEventCreate(&e));
      ev.push_back(e);
    }
  }
  // begin/end of a public call: device time of everything on the stream
  void call_begin() {
    events();
    st.iters = 0;
    st.steps_ms = 0.0;
    st.ms = 0.0;
    PCK(cudaEventRecord(call_ev[0], s));
  }
  void call_end() {
    PCK(cudaEventRecord(call_ev[1], s));
    PCK(cudaEventSynchronize(call_ev[1]));
    float ms = 0.f;
    PCK(cudaEventElapsedTime(&ms, call_ev[0], call_ev[1]));
    st.ms = ms;
    st.kernel_launches = n_launch;
  }
  uint32_t grid() const { return (uint32_t)nsm * 8; }
  // One wave: every block resident at once, so the grid-stride split of the
  // work items has no second partial wave.
  std::map<const void *, uint32_t> rgrid_cache;
  uint32_t rgrid(const void *f) {
    auto it = rgrid_cache.find(f);
    if (it != rgrid_cache.end()) return it->second;
    int b = 0;
    PCK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, f, THREADS, 0));
    const uint32_t g = (uint32_t)nsm * (uint32_t)std::max(b, 1);
    rgrid_cache[f] = g;
    return g;
  }
  void sync() { PCK(cudaStreamSynchronize(s)); }
  // algorithmic bytes of one Jacobi step with K columns: per edge the 4-B
  // neighbour id, the 8-B probability and the neighbour's 8K-B row; per
  // vertex two 8-B offsets and 8K B each of B and x read and out written
  double step_bytes(uint32_t K) const {
    return (double)ne * (12.0 + 8.0 * K) + (double)nv * (16.0 + 24.0 * K);
  }
  cudaMemcpyKind kin(int mem) const {
    return mem == SGS_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  }
  cudaMemcpyKind kout(int mem) const {
    return mem == SGS_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
  }

  void pieces(Adj &a, const uint64_t *ptr, const uint32_t *nbr) {
    a.ptr = ptr;
    a.nbr = nbr;
    a.poff.ensure((size_t)nv + 1);
    { ++n_launch; k_piece_count<<<grid(), THREADS, 0, s>>>(ptr, nv, piece, a.poff.p); }
    size_t tb = 0;
    PCK(cub::DeviceScan::ExclusiveSum(nullptr, tb, a.poff.p, a.poff.p, (int)(nv + 1), s));
    Buf<unsigned char> tmp;
    tmp.ensure(tb);
    PCK(cub::DeviceScan::ExclusiveSum(tmp.p, tb, a.poff.p, a.poff.p, (int)(nv + 1), s));
    PCK(cudaMemcpyAsync(&a.npieces, a.poff.p + nv, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    sync();
    a.pv.ensure(a.npieces);
    { ++n_launch; k_piece_fill<<<grid(), THREADS, 0, s>>>(a.poff.p, nv, a.pv.p); }
    PCK(cudaGetLastError());
  }

  void build(uint32_t n, const uint64_t *r, const uint32_t *c, int mem) {
    nv = n;
    row.ensure((size_t)nv + 1);
    PCK(cudaMemcpyAsync(row.p, r, sizeof(uint64_t) * (nv + 1), kin(mem), s));
    PCK(cudaMemcpyAsync(&ne, row.p + nv, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    sync();
    if (ne >= (1ull << 31)) throw PprFail{SGS_ERR_INVALID, "more than 2^31-1 edges"};
    col.ensure(ne);
    if (ne) PCK(cudaMemcpyAsync(col.p, c, sizeof(uint32_t) * ne, kin(mem), s));
    err.ensure(1);
    PCK(cudaMemsetAsync(err.p, 0, sizeof(unsigned int), s));
    { ++n_launch; k_validate<<<grid(), THREADS, 0, s>>>(row.p, col.p, nv, ne, err.p); }
    unsigned int h = 0;
    PCK(cudaMemcpyAsync(&h, err.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    sync();
    if (h & 2u) throw PprFail{SGS_ERR_INVALID, "row offsets must start at 0 and not decrease"};
    if (h & 1u) throw PprFail{SGS_ERR_INVALID, "column index out of range"};
    // CSC: sort (destination, CSR edge index) by destination (stable, so the
    // in-edges of a vertex keep CSR order), sources through the edge index.
    {
      csrc.ensure(ne);
      ceid.ensure(ne);
      crow.ensure((size_t)nv + 1);
      int bits = 1;
      while (bits < 32 && (1ull << bits) < nv) ++bits;
      size_t tb = 0;
      PCK(cub::DeviceRadixSort::SortPairs(nullptr, tb, col.p, col.p, col.p, ceid.p, (int)ne, 0, bits, s));
      // source, sorted destination and index of every edge, and the sort's
      // storage: one allocation (each costs about as much as a small sort)
      const size_t part3 = (ne * sizeof(uint32_t) + 255) / 256 * 256;
      Buf<unsigned char> tmp;
      tmp.ensure(3 * part3 + tb);
      uint32_t *src = (uint32_t *)tmp.p, *dst_s = (uint32_t *)(tmp.p + part3), *eid = (uint32_t *)(tmp.p + 2 * part3);
      { ++n_launch; k_edge_src<<<grid(), THREADS, 0, s>>>(row.p, nv, src); }
      { ++n_launch; k_iota<<<grid(), THREADS, 0, s>>>(eid, ne); }
      PCK(cub::DeviceRadixSort::SortPairs(tmp.p + 3 * part3, tb, col.p, dst_s, eid, ceid.p, (int)ne, 0, bits, s));
      { ++n_launch; k_csc_rows<<<grid(), THREADS, 0, s>>>(dst_s, ne, nv, crow.p); }
      { ++n_launch; k_gather_u32<<<grid(), THREADS, 0, s>>>(src, ceid.p, ne, csrc.p); }
      PCK(cudaGetLastError());
      sync();
    }
    piece = ne <= SMALL_EDGES ? PIECE_SMALL : PIECE_MAX;
    pieces(in, crow.p, csrc.p);
    pieces(out, row.p, col.p);
    inv_s.ensure(nv);
    pr.ensure(ne);
    pc.ensure(ne);
    const size_t words = 1 + (size_t)std::max(in.npieces, out.npieces);
    work.ensure(sgs::StepHist::FIELDS * (size_t)HIST + (HIST + words + 1) / 2);
    PCK(cudaMemsetAsync(ran(), 0, sizeof(uint32_t) * words, s));
    sync();
  }

  // Loads a weight vector and forms inv_s and the probabilities of the direction
  // asked for: pc (CSC order, forward) or pr (CSR order, adjoint).
  void set_weights(const double *wt, bool adjoint, int mem) {
    w.ensure(ne);
    part.ensure(out.npieces);
    if (ne) PCK(cudaMemcpyAsync(w.p, wt, sizeof(double) * ne, kin(mem), s));
    PCK(cudaMemsetAsync(err.p, 0, sizeof(unsigned int), s));
    { ++n_launch; k_row_sums<<<grid(), THREADS, 0, s>>>(row.p, nv, w.p, out.pv.p, out.poff.p, out.npieces, piece, part.p,
                                                        done(), inv_s.p, adjoint ? pr.p : nullptr, err.p); }
    if (!adjoint)
      { ++n_launch; k_csc_probs<<<grid(), THREADS, 0, s>>>(w.p, inv_s.p, ceid.p, csrc.p, ne, pc.p); }
    else if (out.npieces)
      { ++n_launch; k_piece_probs<<<grid(), THREADS, 0, s>>>(row.p, w.p, out.pv.p, out.poff.p, out.npieces, piece,
                                                             inv_s.p, pr.p); }
    PCK(cudaGetLastError());
    unsigned int h = 0;
    PCK(cudaMemcpyAsync(&h, err.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    sync();
    if (h) throw PprFail{SGS_ERR_INVALID, "edge weights must be positive and finite"};
  }

  template <int L, int C>
  void launch_grad(uint32_t K, double alpha, const double *Y, double *dst) {
    PCK(cudaMemsetAsync(next(), 0, sizeof(uint32_t), s));
    { ++n_launch; k_ppr_edge_grad<L, C><<<rgrid((const void *)k_ppr_edge_grad<L, C>), THREADS, 0, s>>>(
        row.p, col.p, inv_s.p, nv, out.pv.p, out.poff.p, out.npieces, piece, K, alpha, x.p, Y, g.p, dst, next()); }
  }

  // A step of fewer bytes than this (step_bytes) takes less than about 20 us
  // and runs in the launch that loops on the device; a longer one hides its
  // launch, takes its items from a counter and gathers through the read-only
  // cache.  Forward and backward, a launch per step against the loop: 2.8
  // against 1.6 ms at 6 MB a step, 3.9 against 2.7 at 40 MB, 9.8 against 16.1
  // at 189 MB, 104 against 157 at 10 GB.
  static constexpr double LOOP_BYTES = 64e6;

  template <int LPE, int CPL>
  void launch(const StepArgs &a, bool loop, double *b0, double *b1, uint32_t k, uint32_t k1, uint32_t under,
              bool first) {
    if (loop) {
      const void *f = (const void *)k_ppr_steps<LPE, CPL, false>;
      StepArgs aa = a;
      uint32_t *r = ran();
      void *args[] = {&aa, &b0, &b1, &k, &k1, &under, &first, &r};
      // no more CTAs than items (idle ones only lengthen the barriers)
      const uint64_t items = a.npieces + ((uint64_t)a.nv + a.per - 1) / a.per;
      const uint64_t need = (items + THREADS / 32 - 1) / (THREADS / 32);
      uint32_t gr = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(rgrid(f), need));
      // More than two CTAs per SM would queue for the history's words (4,096
      // vertices, K = 32, 512 CTAs: 8.3 us a step with a thread each reading
      // them, 12.0 with all; K = 8, 128 CTAs: 8.5 against 6.5).  Not with 16 lanes
      // per row, where R-MAT graphs' hubs wait for the later start (2^14 vertices,
      // K = 16, forward and backward: 1.66 against 1.57 ms).
      if constexpr (LPE != 16)
        if (gr > 2u * (uint32_t)nsm) {
          f = (const void *)k_ppr_steps<LPE, CPL, true>;
          gr = std::min(gr, rgrid(f));
        }
      ++n_launch;
      PCK(cudaLaunchCooperativeKernel(f, gr, THREADS, args, 0, s));
      return;
    }
    for (; k < k1; ++k) {
      ++n_launch;
      k_ppr_step<LPE, CPL><<<rgrid((const void *)k_ppr_step<LPE, CPL>), THREADS, 0, s>>>(a, k % 2 ? b1 : b0,
                                                                                       k % 2 ? b0 : b1, k, first);
      first = false;
    }
  }
  // Steps k .. k1 - 1 (or, looping, up to the end of the iteration).
  void steps(const StepArgs &a, bool loop, double *b0, double *b1, uint32_t k, uint32_t k1, uint32_t under,
             bool first) {
    switch (a.K <= 32 ? lanes_per_edge(a.K) : 64) {
      case 1: launch<1, 1>(a, loop, b0, b1, k, k1, under, first); break;
      case 2: launch<2, 1>(a, loop, b0, b1, k, k1, under, first); break;
      case 4: launch<4, 1>(a, loop, b0, b1, k, k1, under, first); break;
      case 8: launch<8, 1>(a, loop, b0, b1, k, k1, under, first); break;
      case 16: launch<16, 1>(a, loop, b0, b1, k, k1, under, first); break;
      case 32: launch<32, 1>(a, loop, b0, b1, k, k1, under, first); break;
      default: launch<32, 2>(a, loop, b0, b1, k, k1, under, first); break;
    }
    PCK(cudaGetLastError());
  }

  // Light vertices per item.  From the counter: 8 with up to 8 columns, where the
  // counter sets the pace of finer ones (2^20 vertices, K = 8: 9.9 ms, 11.5 with
  // 4), and with 16 from 2^20 vertices on (12.5 ms, 13.1 with 4); 4 with more (K = 64: 24.0 ms, 24.4 with 8 and 26.0 with 2; 2^18 vertices, K =
  // 16: 4.1 and 4.4 with 8), which keeps the last items short; 2 where a warp gets
  // few items (20,480 vertices, a fifth with 64 edges, K = 64: 8.9 ms, 10.3 with 4 and
  // 12.6 with 8).  In the loop as many as give every warp one item.  At least what
  // the lane groups of a narrow form take at a time, at most 32.
  uint32_t items_per_warp(bool loop, uint32_t K) const {
    const uint32_t warps = (uint32_t)nsm * 32, neg = 32u / (uint32_t)lanes_per_edge(std::min(K, 32u));
    uint32_t per = loop ? (nv + warps - 1) / warps : neg >= 4 || (neg == 2 && nv >= 1u << 20) ? 8u : nv < 8 * warps ? 2u : 4u;
    return std::min(32u, std::max(per, neg));
  }

  // The fixed point of x = c B + alpha A x from c B, in the buffers b0 and b1:
  // steps until one changes the state by less than tol in L1 (ppr_ends).
  // `cur` = the buffer with the result.  Returns the steps run, -1 when max_iter
  // did not suffice: plain steps alone are tried too before that is said, since
  // a long step may fall on the last one permitted, or not keep its promise.
  int iterate(const Adj &adj, const double *p, uint32_t K, double alpha, double c, const double *B, double *b0,
              double *b1, double tol, uint32_t max_iter, double *&cur) {
    bool longs = false;
    st.iters = 0;
    const int it = run_steps(adj, p, K, alpha, c, B, b0, b1, tol, max_iter, false, cur, longs);
    return it >= 0 || !longs ? it : run_steps(adj, p, K, alpha, c, B, b0, b1, tol, max_iter, true, cur, longs);
  }
  int run_steps(const Adj &adj, const double *p, uint32_t K, double alpha, double c, const double *B, double *b0,
                double *b1, double tol, uint32_t max_iter, bool plain, double *&cur, bool &longs) {
    const double bytes = step_bytes(K);
    const bool loop = bytes < LOOP_BYTES;
    StepArgs a{adj.ptr, adj.nbr, p, nv, adj.pv.p, adj.poff.p, adj.npieces, piece, K, alpha, c, B, part.p, done(), next(),
               items_per_warp(loop, K), sgs::StepHist{work.p, HIST}, tol};
    const size_t row = sizeof(double);
    PCK(cudaMemsetAsync(work.p, 0, row * sgs::StepHist::FIELDS * HIST + sizeof(uint32_t) * HIST, s));
    { ++n_launch; k_scale<<<grid(), THREADS, 0, s>>>(B, c, (uint64_t)nv * K, b0); }
    cur = b0;
    uint32_t it = 0, k = 0, under = 0;
    if (plain) {  // after a failed long step none follows
      static const double failed = sgs::ST_FAILED;
      k = 2;
      PCK(cudaMemcpyAsync(sgs::StepHist{work.p, HIST}.state() + 1, &failed, row, cudaMemcpyHostToDevice, s));
    }
    bool below = false;  // a plain step was below tol, and no long one came after it
    double prev = 0.0;   // the last plain step's change
    double norm = 0.0;   // the last step's, whatever its length
    const double entries = (double)nv * K;
    std::vector<double> hd;
    const uint32_t few = bytes > 256e6 ? 2 : 4;
    uint32_t ahead = few;
    while (it < max_iter) {
      if (k == HIST) {
        // the rule looks back four entries: move them to the front.  (An even
        // number, so that k % 2 still names the buffer to read.)
        constexpr uint32_t keep = 4;
        for (int f = 0; f < sgs::StepHist::FIELDS; ++f) {
          double *q = work.p + (size_t)f * HIST;
          PCK(cudaMemcpyAsync(q, q + HIST - keep, row * keep, cudaMemcpyDeviceToDevice, s));
          PCK(cudaMemsetAsync(q + keep, 0, row * (HIST - keep), s));
        }
        PCK(cudaMemsetAsync(next(), 0, sizeof(uint32_t) * HIST, s));
        k = keep;
      }
      // A launch per step: 8 steps before the first host read (never fewer are
      // needed), then 2 to 4 -- a read costs about 10 us, steps past the end
      // their own time -- or, when no long step was taken by step 32, as many as
      // the end is away.
      uint32_t nb = std::min<uint32_t>(HIST - k, max_iter - it);
      if (!loop) nb = std::min<uint32_t>(nb, it == 0 ? 8 : ahead);
      if (timing) PCK(cudaEventRecord(ev[0], s));
      steps(a, loop, b0, b1, k, k + nb, under, it == 0);
      if (timing) PCK(cudaEventRecord(ev[1], s));
      hd.resize(sgs::StepHist::FIELDS * (size_t)nb);
      uint32_t n = nb;
      PCK(cudaMemcpy2DAsync(hd.data(), row * nb, work.p + k, row * HIST, row * nb, sgs::StepHist::FIELDS,
                            cudaMemcpyDeviceToHost, s));
      if (loop) PCK(cudaMemcpyAsync(&n, ran(), sizeof(n), cudaMemcpyDeviceToHost, s));
      sync();
      if (n > nb) throw PprFail{SGS_ERR_CUDA, "PPR step kernel returned a bad step count"};
      if (timing) {
        float ms = 0.f;
        PCK(cudaEventElapsedTime(&ms, ev[0], ev[1]));
        st.steps_ms += ms;
      }
      const sgs::StepHist h{hd.data(), nb};
      // Vertices without edges have their say in step 0 only; one that is not a
      // number there never comes to rest.
      const bool lost = it == 0 && !(h.l1()[0] == h.l1()[0]);
      bool end = false;
      for (uint32_t b = 0; b < n; ++b) {
        const double l1 = h.l1()[b] + sgs::exact_slack(sgs::exact_unit(norm), entries);
        end = end || ppr_ends(h.step()[b], l1, prev, (int)h.state()[b], tol, alpha, under);
        norm = h.l1()[b];
        prev = h.step()[b] == 1.0 ? norm : 0.0;
        below = h.step()[b] == 1.0 && (below || l1 < tol);
        longs = longs || h.step()[b] != 1.0;
      }
      it += n;
      k += n;
      st.iters += (int32_t)n;
      cur = k % 2 ? b1 : b0;
      if (!longs && it >= 32 && n > 1)
        ahead = sgs::StepRule::steps_left(h.l1()[n - 1], h.l1()[n - 2], tol * sgs::LONG_TOL, few, 32);
      else
        ahead = few;
      if (lost) return -1;
      if (end) return (int)it;
    }
    return below ? (int)it : -1;
  }

  int forward(const double *T, uint32_t K, double alpha, double tol, uint32_t max_iter, double *X,
              int mem) {
    const uint64_t n = (uint64_t)nv * K;
    t.ensure(n);
    x.ensure(n);
    xn.ensure(n);
    part.ensure((uint64_t)std::max(in.npieces, out.npieces) * K);
    PCK(cudaMemcpyAsync(t.p, T, sizeof(double) * n, kin(mem), s));
    double *cur = x.p;
    const int it = iterate(in, pc.p, K, alpha, 1.0 - alpha, t.p, x.p, xn.p, tol, max_iter, cur);
    PCK(cudaMemcpyAsync(X, cur, sizeof(double) * n, kout(mem), s));
    sync();
    return it;
  }

  int backward(const double *X, const double *G, uint32_t K, double alpha, double tol,
               uint32_t max_iter, double *gw, double *gT, int mem) {
    const uint64_t n = (uint64_t)nv * K;
    x.ensure(n);
    g.ensure(n);
    y.ensure(n);
    yn.ensure(n);
    part.ensure((uint64_t)std::max(in.npieces, out.npieces) * K);
    PCK(cudaMemcpyAsync(x.p, X, sizeof(double) * n, kin(mem), s));
    PCK(cudaMemcpyAsync(g.p, G, sizeof(double) * n, kin(mem), s));
    double *cur = y.p;
    const int it = iterate(out, pr.p, K, alpha, 1.0, g.p, y.p, yn.p, tol, max_iter, cur);
    if (it < 0) return it;
    if (gw && ne) {
      Buf<double> tmp;
      double *dst = gw;
      if (mem == SGS_MEM_HOST) {
        tmp.ensure(ne);
        dst = tmp.p;
      }
      switch (lanes_per_edge(K)) {
        case 1: launch_grad<1, 1>(K, alpha, cur, dst); break;
        case 2: launch_grad<2, 1>(K, alpha, cur, dst); break;
        case 4: launch_grad<4, 1>(K, alpha, cur, dst); break;
        case 8: launch_grad<8, 1>(K, alpha, cur, dst); break;
        case 16: launch_grad<16, 1>(K, alpha, cur, dst); break;
        default:
          if (K <= 32) launch_grad<32, 1>(K, alpha, cur, dst);
          else launch_grad<32, 2>(K, alpha, cur, dst);
          break;
      }
      PCK(cudaGetLastError());
      if (mem == SGS_MEM_HOST) PCK(cudaMemcpyAsync(gw, dst, sizeof(double) * ne, kout(mem), s));
      sync();
    }
    if (gT) {
      Buf<double> tmp;
      double *dst = gT;
      if (mem == SGS_MEM_HOST) {
        tmp.ensure(n);
        dst = tmp.p;
      }
      { ++n_launch; k_scale<<<grid(), THREADS, 0, s>>>(cur, 1.0 - alpha, n, dst); }
      PCK(cudaGetLastError());
      if (mem == SGS_MEM_HOST) PCK(cudaMemcpyAsync(gT, dst, sizeof(double) * n, kout(mem), s));
      sync();
    }
    sync();
    return it;
  }
};

template <class F>
static int pguard(F &&f) {
  try {
    f();
    return SGS_OK;
  } catch (const PprFail &e) {
    sgs::set_last_error(e.msg);
    return e.code;
  } catch (const std::bad_alloc &) {
    sgs::set_last_error("host allocation failed");
    return SGS_ERR_OOM;
  }
}

static bool bad_args(double alpha, uint32_t K) {
  if (!(alpha > 0.0 && alpha < 1.0)) {
    sgs::set_last_error("alpha must be in (0, 1)");
    return true;
  }
  if (K == 0) {
    sgs::set_last_error("K must be at least 1");
    return true;
  }
  return false;
}

extern "C" {

SGS_API int sgs_ppr_create_csr(int device, uint32_t nv, const uint64_t *row, const uint32_t *col,
                               int mem, sgs_ppr **out) {
  if (!out || !row || !col) {
    sgs::set_last_error("null argument");
    return SGS_ERR_INVALID;
  }
  *out = nullptr;
  if (nv == 0) {
    sgs::set_last_error("empty graph");
    return SGS_ERR_INVALID;
  }
  return pguard([&] {
    auto p = std::make_unique<sgs_ppr>();
    p->dev = device;
    PCK(cudaSetDevice(device));
    PCK(cudaDeviceGetAttribute(&p->nsm, cudaDevAttrMultiProcessorCount, device));
    PCK(cudaStreamCreateWithFlags(&p->s, cudaStreamNonBlocking));
    p->build(nv, row, col, mem);
    *out = p.release();
  });
}

SGS_API int sgs_ppr_create(sgs_engine *e, sgs_ppr **out) {
  if (!e || !out) {
    sgs::set_last_error("null argument");
    return SGS_ERR_INVALID;
  }
  sgs_engine_stats st;
  int rc = sgs_get_engine_stats(e, &st);
  if (rc) return rc;
  std::vector<uint64_t> row((size_t)st.nv + 1);
  std::vector<uint32_t> col(std::max<uint64_t>(st.ne, 1));
  // the export leaves the engine's device current
  rc = sgs_graph_export(e, row.data(), col.data(), nullptr, SGS_MEM_HOST);
  if (rc) return rc;
  int dev = 0;
  cudaGetDevice(&dev);
  return sgs_ppr_create_csr(dev, (uint32_t)st.nv, row.data(), col.data(), SGS_MEM_HOST, out);
}

SGS_API int sgs_ppr_destroy(sgs_ppr *p) {
  if (p) {
    cudaSetDevice(p->dev);
    cudaStreamSynchronize(p->s);
    delete p;
  }
  return SGS_OK;
}

SGS_API int sgs_ppr_info(sgs_ppr *p, uint32_t *nv, uint64_t *ne) {
  if (!p || !nv || !ne) {
    sgs::set_last_error("null argument");
    return SGS_ERR_INVALID;
  }
  *nv = p->nv;
  *ne = p->ne;
  return SGS_OK;
}

SGS_API int sgs_ppr_timing(sgs_ppr *p, int enable) {
  if (!p) {
    sgs::set_last_error("null argument");
    return SGS_ERR_INVALID;
  }
  p->timing = enable != 0;
  return SGS_OK;
}

SGS_API int sgs_ppr_get_stats(sgs_ppr *p, sgs_ppr_stats *out) {
  if (!p || !out) {
    sgs::set_last_error("null argument");
    return SGS_ERR_INVALID;
  }
  p->st.pieces_in = p->in.npieces;
  p->st.pieces_out = p->out.npieces;
  p->st.kernel_launches = p->n_launch;
  *out = p->st;
  return SGS_OK;
}

SGS_API int sgs_ppr_export(sgs_ppr *p, uint64_t *row, uint32_t *col, int mem) {
  if (!p || !row || !col) {
    sgs::set_last_error("null argument");
    return SGS_ERR_INVALID;
  }
  return pguard([&] {
    PCK(cudaSetDevice(p->dev));
    PCK(cudaMemcpyAsync(row, p->row.p, sizeof(uint64_t) * (p->nv + 1), p->kout(mem), p->s));
    if (p->ne) PCK(cudaMemcpyAsync(col, p->col.p, sizeof(uint32_t) * p->ne, p->kout(mem), p->s));
    p->sync();
  });
}

SGS_API int sgs_ppr_forward(sgs_ppr *p, const double *w, const double *T, uint32_t K, double alpha,
                            double tol, uint32_t max_iter, double *X, int *iters, int mem) {
  if (!p || !w || !T || !X) {
    sgs::set_last_error("null argument");
    return SGS_ERR_INVALID;
  }
  if (bad_args(alpha, K)) return SGS_ERR_INVALID;
  return pguard([&] {
    PCK(cudaSetDevice(p->dev));
    p->set_weights(w, false, mem);
    p->call_begin();
    p->st.bytes_alg_step = p->step_bytes(K);
    const int it = p->forward(T, K, alpha, tol, max_iter, X, mem);
    p->call_end();
    if (iters) *iters = it;
    if (it < 0) throw PprFail{SGS_ERR_NOCONV, "PPR forward did not converge"};
  });
}

SGS_API int sgs_ppr_backward(sgs_ppr *p, const double *w, const double *X, const double *G,
                             uint32_t K, double alpha, double tol, uint32_t max_iter, double *gw,
                             double *gT, int *iters, int mem) {
  if (!p || !w || !X || !G) {
    sgs::set_last_error("null argument");
    return SGS_ERR_INVALID;
  }
  if (bad_args(alpha, K)) return SGS_ERR_INVALID;
  return pguard([&] {
    PCK(cudaSetDevice(p->dev));
    p->set_weights(w, true, mem);
    p->call_begin();
    p->st.bytes_alg_step = p->step_bytes(K);
    const int it = p->backward(X, G, K, alpha, tol, max_iter, gw, gT, mem);
    p->call_end();
    if (iters) *iters = it;
    if (it < 0) throw PprFail{SGS_ERR_NOCONV, "PPR adjoint did not converge"};
  });
}

}  // extern "C"
