"""Branches that depend on a graph's size or shape, at their edges:

* the repair of a narrow group after deletions: nothing reset, few vertices
  reset (restricted sweep), more than half of them (full sweep); the
  sweep's filter exact (up to 2^20 vertices) and folded (above), blocks below
  and above its slice sizes, the last vertex reset, host tier and cache;
* the batch sort at the edges of a vertex id's bits, with inserts only,
  deletes only and inserts that the same batch deletes;
* step lengths: PageRank and PPR on graphs with and without a spectral gap;
* PageRank's absorb with one and with four vertices per thread;
* PPR in the looping launch and in a launch per step, with light vertices and
  pieces of either size;
* results gathered by several threads at once.
"""
import threading

import numpy as np
import pytest

import oracle as O
import ppr_dense as D
import sgs
from test_gpu_parity import Mirror, check_graph, check_query

pytestmark = pytest.mark.gpu

ALPHA = 0.85


def _load(nv, src, dst, seed=1, **cfg):
    row, col = O.csr_from_edges(nv, np.asarray(src, np.uint32), np.asarray(dst, np.uint32))
    w = O.weights(nv, row, col, seed, 0)
    e = sgs.Engine(**cfg)
    e.load_csr(nv, row, col, w)
    return e, Mirror(nv, row, col, w)


def _apply(e, m, ins, dele, seed=1):
    i_s, i_d = (np.asarray(a, np.uint32) for a in ins)
    d_s, d_d = (np.asarray(a, np.uint32) for a in dele)
    w = O.weights_pairs(seed, i_s, i_d) if len(i_s) else np.empty(0, np.uint32)
    e.apply_batch(i_s, i_d, w, d_s, d_d)
    m.apply(i_s, i_d, w, d_s, d_d)


def _hub_graph(nv, hub_degree, seed):
    """A hub (vertex 0) of the given degree, a chain through the last vertices
    and random edges."""
    rng = np.random.default_rng(seed)
    n = min(4 * nv, 6000)
    out = rng.choice(np.arange(1, nv), hub_degree, replace=False)
    tail = np.arange(max(1, nv - 40), nv - 1)
    src = np.concatenate([np.zeros(hub_degree, np.int64), tail, rng.integers(0, nv, n)])
    dst = np.concatenate([out, tail + 1, rng.integers(0, nv, n)])
    return src, dst


@pytest.mark.parametrize("tier", ["hbm", "host"])
@pytest.mark.parametrize("nv,hub", [(300, 256), (2000, 257), (4000, 1025), ((1 << 20) + 33, 5000)])
def test_repair_modes(nv, hub, tier):
    cfg = {} if tier == "hbm" else dict(hbm_budget_gb=2e-5, cache_gb=1e-5, segments=16)
    e, m = _load(nv, *_hub_graph(nv, hub, nv), **cfg)
    with e:
        qs = e.add_queries([(sgs.SSSP, 0), (sgs.BFS, 0), (sgs.CC, 0), (sgs.SSSP, nv - 40)])

        def check():
            for q in qs:
                check_query(q, m, sgs.W_EXPLICIT)

        # edges into the last vertex and a few of the hub's: some resets
        par = qs[1].parent()
        some = [nv - 1] + [int(v) for v in m.col[m.row[0]:m.row[0] + 5]]
        some = [(int(par[v]), v) for v in some if par[v] != sgs.INF]
        _apply(e, m, ([], []), ([u for u, _ in some], [v for _, v in some]))
        assert qs[1].stats()["invalidated"] >= len(some) > 0
        check()
        # a non-tree edge, if there is one: no reset, inserts alone
        par = qs[0].parent(), qs[1].parent(), qs[2].parent(), qs[3].parent()
        src = np.repeat(np.arange(nv), np.diff(m.row).astype(np.int64))
        free = np.nonzero(np.all([p[m.col] != src for p in par], axis=0))[0][:3]
        _apply(e, m, ([5, 6], [nv - 1, nv - 2]), (src[free], m.col[free]))
        assert all(q.stats()["invalidated"] == 0 for q in qs)
        check()
        # every edge of the hub: most of the graph is reset (full sweep on the
        # small ones), and some of it comes back another way
        u0, u1 = int(m.row[0]), int(m.row[1])
        hubs = m.col[u0:u1].copy()
        _apply(e, m, (np.zeros(4), [7, 8, 9, nv - 3]), (np.zeros(len(hubs)), hubs))
        check()
        # and back
        _apply(e, m, (np.zeros(len(hubs)), hubs), ([0, 0], [7, 8]))
        check()
        if nv <= 4000:
            check_graph(e, m)


@pytest.mark.parametrize("nv", [2, 3, 255, 256, 257, 1023, 1025])
def test_batch_sort_id_edges(nv):
    rng = np.random.default_rng(nv)
    e, m = _load(nv, rng.integers(0, nv, 4 * nv), rng.integers(0, nv, 4 * nv))
    with e:
        q = e.add_query(sgs.SSSP, nv - 1)
        top = nv - 1
        batches = [
            (([top, 0, top], [0, top, 1]), ([], [])),          # inserts only
            (([], []), ([top, 0], [0, top])),                  # deletes only
            (([top, 0, 0], [0, top, 1]), ([0], [top])),        # one insert deleted again
            (([0, 1 % nv], [top, top]), ([0, 1 % nv], [top, top])),  # all of them
        ]
        for ins, dele in batches:
            keep = [k for k in range(len(ins[0])) if ins[0][k] != ins[1][k]]
            ins = ([ins[0][k] for k in keep], [ins[1][k] for k in keep])
            _apply(e, m, ins, dele)
            check_graph(e, m)
            check_query(q, m, sgs.W_EXPLICIT)


def _shapes():
    n = 600
    rng = np.random.default_rng(3)
    a = np.arange(n)
    half = n // 2
    return {
        "cycle": (n, a, (a + 1) % n),
        "star": (n, np.concatenate([a[1:], np.zeros(n - 1)]), np.concatenate([np.zeros(n - 1), a[1:]])),
        "path": (n, np.concatenate([a[:-1], a[1:]]), np.concatenate([a[1:], a[:-1]])),
        "bipartite": (n, np.concatenate([np.repeat(a[:half], 4), np.repeat(a[half:], 4)]),
                      np.concatenate([rng.integers(half, n, 4 * half), rng.integers(0, half, 4 * half)])),
        "two parts": (n, np.concatenate([rng.integers(0, half, 2000), rng.integers(half, n, 900)]),
                      np.concatenate([rng.integers(0, half, 2000), rng.integers(half, n, 900)])),
        "no edges": (n, [], []),
    }


@pytest.mark.parametrize("pull,persistent", [(1, 14), (1, 6), (0, 14)])
@pytest.mark.parametrize("shape", list(_shapes()))
def test_pagerank_step_lengths(shape, pull, persistent):
    """The documented stop rule (sum of residuals below 1.5e-7) bounds the
    L-infinity error by 1e-6 on any graph, after a start and an update."""
    nv, src, dst = _shapes()[shape]
    e, m = _load(nv, src, dst, pull=pull, persistent=persistent)
    with e:
        q = e.add_query(sgs.PR)
        check_query(q, m, sgs.W_EXPLICIT)
        for k in range(2):
            d = np.arange(k, len(m.col), 7)[:20]
            u = np.repeat(np.arange(nv), np.diff(m.row).astype(np.int64))[d]
            _apply(e, m, ([1, 2, nv - 1], [nv - 1, 5 + k, 0]), (u, m.col[d]))
            check_query(q, m, sgs.W_EXPLICIT)


@pytest.mark.parametrize("nv", [1184 * 1024, 1184 * 1024 + 1, 1184 * 2048 - 1])
@pytest.mark.parametrize("pull", [0, 1])
def test_pagerank_absorb_widths(nv, pull):
    """Sizes around the one from which an absorb launch takes four vertices per
    thread at a time (more than four for each of 1184 * 256 threads)."""
    rng = np.random.default_rng(nv)
    src, dst = rng.integers(0, nv, (2, 30000))
    tail = np.arange(nv - 300, nv - 1)
    e, m = _load(nv, np.concatenate([src, tail]), np.concatenate([dst, tail + 1]), pull=pull, persistent=6)
    with e:
        q = e.add_query(sgs.PR)
        check_query(q, m, sgs.W_EXPLICIT)
        _apply(e, m, ([nv - 1, 0], [0, nv - 1]), (tail[::7], tail[::7] + 1))
        check_query(q, m, sgs.W_EXPLICIT)


@pytest.mark.parametrize("K", [1, 2, 16, 17, 65])
@pytest.mark.parametrize("shape", [s for s in _shapes() if s != "no edges"])
def test_ppr_step_lengths(shape, K):
    """Forward and adjoint against the dense solve: the L1 error is at most
    alpha / (1 - alpha) times the last step's change, which is below tol."""
    nv, src, dst = _shapes()[shape]
    row, col = O.csr_from_edges(nv, np.asarray(src, np.uint32), np.asarray(dst, np.uint32))
    rng = np.random.default_rng(K)
    w = np.exp(rng.uniform(-2, 2, len(col)))
    T = np.zeros((nv, K))
    T[rng.integers(0, nv, 4 * K), rng.integers(0, K, 4 * K)] = 1.0
    G = rng.standard_normal((nv, K))
    tol = 1e-13 * nv * K
    with sgs.Ppr(nv, row, col) as g:
        X = g.forward(w, T, tol=tol)
        gw, gT = g.backward(w, X, G, tol=tol)
    ref = D.ppr_dense(nv, row, col, w, T)
    assert np.abs(X - ref).sum() <= 6 * tol
    _, rw, rT = D.ppr_grad_closed(nv, row, col, w, T, G)
    # the adjoint's matrix has row sums alpha, so its error is at most 6 tol
    # anywhere; dw_uv = X[u] . (alpha Y[v] - Y[u] + G[u]) / s_u
    Y = rT / (1 - ALPHA)
    assert np.max(np.abs(gT - rT)) <= (1 - ALPHA) * 6 * tol + 1e-13 * np.abs(rT).max()
    s = np.bincount(np.repeat(np.arange(nv), np.diff(row).astype(np.int64)), weights=w, minlength=nv)
    bound = (6 * tol * (2 * np.abs(Y).max() + np.abs(G).max()) + 12 * tol * ref.sum(1).max()) / s[s > 0].min()
    assert np.max(np.abs(gw - rw)) <= bound + 1e-12 * np.abs(rw).max()


@pytest.mark.parametrize("K", [1, 8, 40])
@pytest.mark.parametrize("scale,ef", [(10, 16), (13, 16), (17, 20)])
def test_ppr_launch_forms(scale, ef, K):
    """Sizes on both sides of the looping launch's limit and of the piece
    sizes' (2^21 edges), against the sparse Jacobi oracle."""
    nv, row, col = O.rmat_csr(scale, ef, 5)
    rng = np.random.default_rng(scale)
    w = np.exp(rng.uniform(-2, 2, len(col)))
    T = np.zeros((nv, K))
    T[rng.integers(0, nv, 32), np.arange(32) % K] = 1.0
    tol = 1e-12
    with sgs.Ppr(nv, row, col) as g:
        X = g.forward(w, T, tol=tol)
    Y = X
    for _ in range(3):  # one more step changes it by less than tol (and rounding)
        Y, _ = D.ppr_jacobi_sparse(nv, row, col, w, T, iters=1, X0=Y)
    assert np.abs(Y - X).sum() <= 6 * tol + 1e-15 * np.abs(X).sum() * 64


def test_gather_from_threads():
    nv, row, col = O.rmat_csr(14, 16, 9)
    w = O.weights(nv, row, col, 1, 0)
    with sgs.Engine() as e:
        e.load_csr(nv, row, col, w)
        qs = e.add_queries([(sgs.SSSP, 0), (sgs.BFS, 0), (sgs.CC, 0)])
        want = [q.value() for q in qs]
        bad = []

        def read(k):
            for _ in range(20):
                if not np.array_equal(qs[k].value(), want[k]):
                    bad.append(k)

        ts = [threading.Thread(target=read, args=(k,)) for k in range(3)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert not bad
