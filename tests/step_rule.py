"""The step lengths of PageRank and PPR on the CPU (test infrastructure): how
many steps plain iteration takes to a tolerance, and where the first long step
falls, so that tests can put a limit right there."""
import numpy as np


def _long_step(hist, alpha, tol):
    """The length of the next step from the norms of the ones before it."""
    if len(hist) < 2:
        return 1.0, 0.0
    (a, f, mu0), (b, _, _) = hist[-1], hist[-2]
    mu = a / b
    if not 0.3 < mu <= alpha * 1.0001 or a < tol:
        return 1.0, 0.0
    if mu0 > 0 and f + abs(mu - mu0) * b < 0.2 * (1 - mu) * a:
        return 1 / (1 - mu), mu
    return 1.0, mu


def first_long_step(M, c, B, alpha, steps=60):
    """Norms of the plain steps x <- c B + alpha M x from c B up to the first
    step k that would be a long one: (k, [|d_0| .. |d_k|])."""
    x = c * B
    prev = np.zeros_like(x)
    hist, norms = [], []
    for k in range(steps):
        w, mu = _long_step(hist, alpha, 0.0)
        d = c * B + alpha * (M @ x) - x
        norms.append(float(np.abs(d).sum()))
        if w != 1.0:
            return k, norms
        hist.append((norms[-1], float(np.abs(d - mu * prev).sum()) if mu else 0.0, mu))
        prev, x = d, x + d
    return None, norms


def first_long_round(M, nv, alpha, has_out, rounds=60):
    """The same for the engine's PageRank, whose round k absorbs the residual
    r_k (r_0 = 1 - alpha everywhere)."""
    r = np.full(nv, 1 - alpha)
    prev = np.zeros(nv)
    hist, norms = [], []
    for k in range(rounds):
        w, mu = _long_step(hist, alpha, 0.0)
        norms.append(float(np.abs(r).sum()))
        if w != 1.0:
            return k, norms
        fit = float(np.abs(r - mu * prev)[has_out].sum()) if mu else 0.0
        hist.append((norms[-1], fit, mu))
        prev, r = r, alpha * (M @ r)
    return None, norms
