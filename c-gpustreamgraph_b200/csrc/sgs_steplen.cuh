// sgs_steplen.cuh -- step lengths of the engine's fixed-point iterations
// (PageRank rounds in sgs_kernels.cuh, personalized PageRank in ppr.cu).
//
// Both iterate x <- x + w d with d = c + M x - x, M = alpha P^T (or alpha P for
// the adjoint): w = 1 is the reference's round.  Whatever the steps were, x is
// that much nearer or further, never wrong: d is the residual of the
// x at hand, and the iteration ends on a plain step whose d is below the
// tolerance.
//
// With w = 1, d shrinks by M's largest eigenvalue mu per step -- 0.84 on R-MAT
// graphs -- while everything in it beside the Perron vector shrinks by the
// second one, 0.15 there.  So after a few steps d is all but a multiple of
// that vector, and one long step, w = 1 / (1 - mu), whose factor
// 1 - w (1 - lambda) is zero at lambda = mu, removes it.
// mu is the ratio of the L1 norms of two successive d.  A long step leaves
// w (d_k+1 - mu d_k), so the steps before it measure that: `fit` is the norm of
// d_k - mu d_k-1 (one more read per vertex), and the long step is taken when it
// would leave less than a fifth of d.  On graphs without such a gap
// (bipartite ones, grids, cycles with a mixed-sign d) the fit stays bad and
// every step stays plain.  Should a long step not halve d after all, no
// other one follows.
// Steps to the tolerance, long steps included, on R-MAT graphs of scale 10 to
// 18: PageRank from scratch 116-151 -> 22-26, after an update 59-85 -> 18-21.
//
// Once a long step was taken, the end asks for a sixteenth of the tolerance
// (one or two steps at the faster rate): the error at the end, 1e-9 to 1e-8 of
// L1 norm instead of 7e-7 in those runs, is then no larger than that of the slow
// approach and the steps that were queued past its end.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace sgs {

enum StepState : int { ST_PLAIN = 0, ST_LONG = 1, ST_FAILED = 2 };
constexpr double LONG_TOL = 1.0 / 16.0;

// One entry per step in device memory, zeroed before the first: |d|, the fit
// and the mu it was taken with (0: none was), the step length (0 marks a d
// that was changed between two steps, so no ratio across it counts), state.
// Fields are `n` entries apart.  A step's rule reads entries that earlier
// launches, or phases before a grid barrier, wrote.
struct StepHist {
  static constexpr int FIELDS = 5;
  double *p;
  uint32_t n;
  __host__ __device__ double *l1() const { return p; }
  __host__ __device__ double *fit() const { return p + n; }
  __host__ __device__ double *mu() const { return p + 2 * (size_t)n; }
  __host__ __device__ double *step() const { return p + 3 * (size_t)n; }
  __host__ __device__ double *state() const { return p + 4 * (size_t)n; }
};

// A sum whose value must not depend on the order of its additions is made of
// exact_terms: x >= 0 rounded to a multiple of 2^-47 of the last step's norm (of
// its power of two, the unit), of which up to 2^53 add up without rounding.  The
// last bit of a number of 48 units' size is such a multiple.  (Unit 0: no norm to
// go by, x is left as it is.)  The sum of n terms is off by exact_slack at most.
__host__ __device__ __forceinline__ double exact_unit(double norm) {
  unsigned long long b;
  memcpy(&b, &norm, sizeof(b));
  b &= 0x7FF0000000000000ull;
  double u;
  memcpy(&u, &b, sizeof(u));
  return u < 1e300 ? u : 0.0;
}
__device__ __forceinline__ double exact_term(double x, double unit) {
  const double c = 48.0 * unit;
  return __dsub_rn(__dadd_rn(x, c), c);
}
__host__ __device__ __forceinline__ double exact_slack(double unit, double n) {
  return n * (unit * (1.0 / (double)(1ull << 48)));
}

struct StepRule {
  // The plain steps that norms falling as the last two did take to tol, in
  // [least, most] (host: how many to queue before the next look).
  static uint32_t steps_left(double l1, double before, double tol, uint32_t least, uint32_t most) {
    if (!(l1 > tol && l1 < before && tol > 0.0)) return least;
    const double n = std::ceil(std::log(l1 / tol) / std::log(before / l1));
    return n > least ? (n < most ? (uint32_t)n : most) : least;
  }
  double w;   // step length
  double mu;  // > 0: take the fit with it
  int state;
  double unit = 0.0;  // exact_term's
  // whether a step with norm l1 under this rule ends the iteration
  __host__ __device__ static bool ends(double w, double l1, int state, double tol) {
    return w == 1.0 && l1 < (state == ST_LONG ? tol * LONG_TOL : tol);
  }
};

// Exact: the norms are sums of exact_terms, so that a step's length, and with it
// the state, is the same to the last bit in equal calls.  (The fit is not: it is
// compared with a threshold only.)
template <bool Exact = false>
__device__ __forceinline__ StepRule step_rule(const StepHist &h, uint32_t k, double alpha, double tol) {
  if (k == 0) return StepRule{1.0, 0.0, ST_PLAIN};
  // (all that may be needed at once: one round trip)
  const uint32_t k1 = k - 1, k2 = k > 1 ? k - 2 : 0, k3 = k > 2 ? k - 3 : 0;
  const double a = __ldcg(h.l1() + k1), b = __ldcg(h.l1() + k2), c = Exact ? __ldcg(h.l1() + k3) : 0.0;
  const double w1 = __ldcg(h.step() + k1), w2 = __ldcg(h.step() + k2);
  const double f = __ldcg(h.fit() + k1), mu0 = __ldcg(h.mu() + k1);
  StepRule s{1.0, 0.0, (int)__ldcg(h.state() + k1)};
  if (Exact) s.unit = exact_unit(a);
  if (k < 2 || s.state == ST_FAILED) return s;
  if (w2 > 1.0 && !(a < 0.5 * b)) {
    s.state = ST_FAILED;
    return s;
  }
  if (w1 != 1.0 || w2 != 1.0 || !(b > 0.0)) return s;
  // (sums of a step whose norm grew more than eightfold may have been rounded)
  if (Exact && k > 2 && !(b <= 8.0 * c)) return s;
  const double mu = a / b;
  // (below 0.3 a plain step is as good; M's spectral radius is at most alpha)
  if (!(mu > 0.3 && mu <= alpha * 1.0001)) return s;
  // no long step near the end: a step queued past it must not raise d
  if (a < (s.state == ST_LONG ? tol * LONG_TOL : tol)) return s;
  s.mu = mu;
  if (mu0 > 0.0 && f + fabs(mu - mu0) * b < 0.2 * (1.0 - mu) * a) {
    s.w = 1.0 / (1.0 - mu);
    s.state = ST_LONG;
  }
  return s;
}

// Records step k's rule (one thread of the step's grid).
__device__ __forceinline__ void record_rule(const StepHist &h, uint32_t k, const StepRule &s) {
  h.mu()[k] = s.mu;
  h.step()[k] = s.w;
  h.state()[k] = (double)s.state;
}

}  // namespace sgs
