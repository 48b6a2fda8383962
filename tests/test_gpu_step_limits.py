"""PPR's and PageRank's iterations at their limits:

* the documented end (one step's L1 change below the tolerance, or the sum of
  the residuals for PageRank) is found within the steps that plain iteration
  needs, also when one of them is a long step;
* input that is not a number is refused wherever it stands;
* two runs give the same bits;
* PPR's launch per step: the adjoint and the edge gradient, all column
  layouts, and more steps than the step history holds, in both launch forms.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle as O
import ppr_dense as D
import sgs
import step_rule as S

pytestmark = pytest.mark.gpu

ALPHA = 0.85
NOCONV = -5


def _p(nv, row, col, w):
    """Row-normalised transition matrix, sparse."""
    src = np.repeat(np.arange(nv), np.diff(row).astype(np.int64))
    s = np.bincount(src, weights=w, minlength=nv)
    return sp.csr_matrix((w / s[src], (src, col.astype(np.int64))), shape=(nv, nv))


def _inputs(nv, ne, K, seed):
    rng = np.random.default_rng(seed)
    T = np.zeros((nv, K))
    T[rng.integers(0, nv, 32), np.arange(32) % K] = 1.0
    return np.exp(rng.uniform(-1, 1, ne)), T, rng.standard_normal((nv, K))


@pytest.mark.parametrize("scale,K", [(8, 1), (10, 3), (12, 20)])
def test_ppr_limit_where_plain_steps_suffice(scale, K):
    """Plain steps are below tol at step k, where the rule takes a long one."""
    nv, row, col = O.rmat_csr(scale, 16, 2)
    w, T, G = _inputs(nv, len(col), K, scale)
    P = _p(nv, row, col, w)
    with sgs.Ppr(nv, row, col) as g:
        k, n = S.first_long_step(P.T.tocsr(), 1 - ALPHA, T, ALPHA)
        assert k is not None and n[k] < n[k - 1]
        tol = 0.5 * (n[k] + n[k - 1])
        X = g.forward(w, T, tol=tol, max_iter=k + 1)
        assert g.last_iters <= k + 1
        # the L1 error is at most alpha / (1 - alpha) times the last change
        assert np.abs(X - D.ppr_dense(nv, row, col, w, T)).sum() <= ALPHA / (1 - ALPHA) * tol
        with pytest.raises(sgs.SgsError) as err:  # one step fewer never was enough
            g.forward(w, T, tol=0.5 * n[-1] * 1e-3, max_iter=3)
        assert err.value.code == NOCONV
        # the adjoint; a positive G has a Perron part, so a long step comes
        k, n = S.first_long_step(P, 1.0, np.abs(G), ALPHA)
        assert k is not None and n[k] < n[k - 1]
        tol = 0.5 * (n[k] + n[k - 1])
        _, gT = g.backward(w, X, np.abs(G), tol=tol, max_iter=k + 1)
        Y = np.linalg.solve(np.eye(nv) - ALPHA * P.toarray(), np.abs(G))
        # row sums of alpha P are at most alpha: the same bound for the maximum
        assert np.abs(gT / (1 - ALPHA) - Y).max() <= ALPHA / (1 - ALPHA) * tol


@pytest.mark.parametrize("pull,persistent", [(1, 14), (1, 6), (0, 14)])
@pytest.mark.parametrize("scale", [8, 11])
def test_pagerank_limit_where_plain_rounds_suffice(scale, pull, persistent):
    nv, row, col = O.rmat_csr(scale, 16, 2)
    P = _p(nv, row, col, np.ones(len(col)))
    k, n = S.first_long_round(P.T.tocsr(), nv, ALPHA, np.diff(row) > 0)
    assert k is not None and n[k] < n[k - 1]
    tol = 0.5 * (n[k] + n[k - 1])
    ref = O.pagerank(nv, row, col)
    with sgs.Engine(max_rounds=k + 1, pr_tol=tol, pull=pull, persistent=persistent) as e:
        e.load_csr(nv, row, col, O.weights(nv, row, col, 1, 0))
        q = e.add_query(sgs.PR)
        assert q.stats()["converged"] == 1 and q.stats()["pr_residual_l1"] < tol
        # what is left after the residual r is at most |r| / (1 - alpha)
        assert np.abs(q.value() - ref).sum() <= ALPHA / (1 - ALPHA) * tol
        e.remove_query(q)
    with sgs.Engine(max_rounds=k + 1, pr_tol=tol, pull=pull, persistent=persistent, pr_warm=0) as e:
        e.load_csr(nv, row, col, O.weights(nv, row, col, 1, 0))
        out = np.empty(nv)
        done = e.serve([{"kind": "query", "algo": sgs.PR, "value_out": out}], realtime=False)
        assert done[0]["status"] == 0
        assert np.abs(out - ref).sum() <= ALPHA / (1 - ALPHA) * tol


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("nv", [50, 1 << 19])
def test_ppr_refuses_what_is_not_a_number(nv, bad):
    """Also at a vertex without any edge, in a launch per step (2^19 vertices,
    K = 8: 109 MB a step) and in the looping launch."""
    K = 8
    a = np.arange(40)
    row, col = O.csr_from_edges(nv, np.concatenate([a, a]).astype(np.uint32),
                                np.concatenate([(a + 1) % 41, (a * 7 + 3) % 41]).astype(np.uint32))
    w = np.ones(len(col))
    T = np.zeros((nv, K))
    T[:41] = 1.0
    with sgs.Ppr(nv, row, col) as g:
        X = g.forward(w, T)
        for v in (5, 45):
            T2 = T.copy()
            T2[v, 3] = bad
            with pytest.raises(sgs.SgsError) as err:
                g.forward(w, T2, max_iter=300)
            assert err.value.code == NOCONV
            with pytest.raises(sgs.SgsError) as err:
                g.backward(w, X, T2, max_iter=300)
            assert err.value.code == NOCONV
        assert np.array_equal(g.forward(w, T), X)


@pytest.mark.parametrize("scale,K", [(12, 8), (13, 40), (17, 8), (17, 40)])
def test_ppr_repeats_itself(scale, K):
    """Equal bits from run to run (torch's gradcheck asks for them), many CTAs,
    both launch forms."""
    nv, row, col = O.rmat_csr(scale, 16, 7)
    w, T, G = _inputs(nv, len(col), K, scale)
    with sgs.Ppr(nv, row, col) as g:
        X = g.forward(w, T)
        gw, gT = g.backward(w, X, G)
        for _ in range(6):
            assert np.array_equal(g.forward(w, T), X)
            gw2, gT2 = g.backward(w, X, G)
            assert np.array_equal(gT2, gT) and np.array_equal(gw2, gw)


@pytest.mark.parametrize("K", [3, 8, 16, 20, 40])
def test_ppr_launch_per_step_adjoint(K):
    """Scale 17, pieces of 128 edges: 64 MB a step or more from K = 3 on."""
    nv, row, col = O.rmat_csr(17, 20, 5)
    w, T, G = _inputs(nv, len(col), K, K)
    P = _p(nv, row, col, w)
    tol = 1e-10
    with sgs.Ppr(nv, row, col) as g:
        X = g.forward(w, T, tol=tol)
        gw, gT = g.backward(w, X, G, tol=tol)
    # one more step changes the states by less than tol, and the rounding of
    # a row's sum
    d = (1 - ALPHA) * T + ALPHA * (P.T @ X) - X
    assert np.abs(d).sum() <= tol + 64 * 1e-15 * np.abs(X).sum()
    Y = gT / (1 - ALPHA)
    d = G + ALPHA * (P @ Y) - Y
    assert np.abs(d).sum() <= tol + 64 * 1e-15 * np.abs(Y).sum()
    # gw_uv = X[u] . (alpha Y[v] - Y[u] + G[u]) / s_u: edges at random and all of
    # the largest row's
    src = np.repeat(np.arange(nv), np.diff(row).astype(np.int64))
    s = np.bincount(src, weights=w, minlength=nv)
    hub = int(np.argmax(np.diff(row)))
    pick = np.concatenate([np.random.default_rng(1).integers(0, len(col), 5000),
                           np.arange(row[hub], row[hub + 1]).astype(np.int64)])
    u, v = src[pick], col[pick].astype(np.int64)
    ref = np.einsum("ek,ek->e", X[u], ALPHA * Y[v] - Y[u] + G[u]) / s[u]
    mag = np.einsum("ek,ek->e", np.abs(X[u]), np.abs(Y[v]) + np.abs(Y[u]) + np.abs(G[u])) / s[u]
    assert np.all(np.abs(gw[pick] - ref) <= 1e-13 * mag)


@pytest.mark.parametrize("nv", [600, 1 << 19])
def test_ppr_more_steps_than_the_history(nv):
    """A cycle at alpha = 0.98 takes some 1,300 steps, all plain; its solution
    is a geometric series."""
    alpha, K = 0.98, 8
    a = np.arange(nv)
    row, col = O.csr_from_edges(nv, a.astype(np.uint32), ((a + 1) % nv).astype(np.uint32))
    T = np.zeros((nv, K))
    T[np.arange(K) * 7, np.arange(K)] = 1.0
    tol = 1e-11
    with sgs.Ppr(nv, row, col) as g:
        X = g.forward(np.ones(nv), T, alpha=alpha, tol=tol)
        assert g.last_iters > 1024
    ref = np.zeros_like(T)
    for k in range(K):
        ref[(np.arange(nv) + 7 * k) % nv, k] = (1 - alpha) * alpha ** np.arange(nv) / (1 - alpha**nv)
    assert np.abs(X - ref).sum() <= alpha / (1 - alpha) * tol


@pytest.mark.parametrize("nv0", [1 << 10, 1 << 17])
def test_ppr_long_steps_and_more_steps_than_the_history(nv0):
    """An R-MAT part, whose Perron vector one long step removes, beside a
    cycle with a thousandth of the mass, which keeps the rest of the steps
    plain and takes more of them than the history holds."""
    alpha, K, ring = 0.98, 4, 3000
    n0, row, col = O.rmat_csr(int(np.log2(nv0)), 16, 3)
    src = np.repeat(np.arange(n0), np.diff(row).astype(np.int64))
    a = np.arange(ring)
    nv = n0 + ring
    row, col = O.csr_from_edges(nv, np.concatenate([src, n0 + a]).astype(np.uint32),
                                np.concatenate([col.astype(np.int64), n0 + (a + 1) % ring]).astype(np.uint32))
    w = np.ones(len(col))
    T = np.zeros((nv, K))
    T[:n0] = 1.0
    T[n0 + np.arange(K), np.arange(K)] = 1e-3 * n0
    tol = 1e-9
    with sgs.Ppr(nv, row, col) as g:
        X = g.forward(w, T, alpha=alpha, tol=tol)
        assert g.last_iters > 512
    P = _p(nv, row, col, w)
    d = (1 - alpha) * T + alpha * (P.T @ X) - X
    assert np.abs(d).sum() <= tol + 64 * 1e-15 * np.abs(X).sum()


@pytest.mark.parametrize("K", [1, 2, 3, 8, 16])
@pytest.mark.parametrize("degree", [32, 33, 60, 64])
def test_ppr_items_of_heavier_vertices(degree, K):
    """Whole items of vertices at and above the 32 edges that a lane group takes
    by itself, and the odd one among lighter ones, up to the piece size of small
    graphs (64)."""
    n = 300
    rng = np.random.default_rng(degree)
    src = [np.argsort(rng.random((n, n)), axis=1)[:, :degree]]  # in-neighbours of [0, n)
    dst = [np.repeat(np.arange(n), degree).reshape(n, degree)]
    light = n + np.arange(700)  # lighter ones, every 50th as heavy
    deg = np.where(light % 50 == 0, degree, 3)
    src.append(rng.integers(0, n + 700, deg.sum()))
    dst.append(np.repeat(light, deg))
    nv = n + 700
    row, col = O.csr_from_edges(nv, np.concatenate([a.ravel() for a in src]).astype(np.uint32),
                                np.concatenate([a.ravel() for a in dst]).astype(np.uint32))
    w, T, G = _inputs(nv, len(col), K, degree)
    tol = 1e-13 * nv * K
    with sgs.Ppr(nv, row, col) as g:
        X = g.forward(w, T, tol=tol)
        gw, gT = g.backward(w, X, G, tol=tol)
    assert np.abs(X - D.ppr_dense(nv, row, col, w, T)).sum() <= ALPHA / (1 - ALPHA) * tol
    Y = np.linalg.solve(np.eye(nv) - ALPHA * _p(nv, row, col, w).toarray(), G)
    assert np.abs(gT / (1 - ALPHA) - Y).max() <= ALPHA / (1 - ALPHA) * tol + 1e-13 * np.abs(Y).max()
