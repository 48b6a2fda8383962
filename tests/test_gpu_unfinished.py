"""Snapshots that end with an error, and the ones after them: a snapshot may
assume that a group's values satisfied every edge before it only if the one
before it was repaired to the end.  After a round limit, a user algorithm's
error or PageRank's round limit, the next snapshot has to bring every query
to its exact result, whatever it inserts and deletes itself.
"""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import sgs
from test_gpu_parity import Mirror, check_query

pytestmark = pytest.mark.gpu

NOCONV = -5
NONE = np.empty(0, np.uint32)


def _weights(src, dst):
    return O.weights_pairs(1, np.asarray(src, np.uint32), np.asarray(dst, np.uint32)) if len(src) else NONE


def _batch(ins, dele):
    i_s, i_d, d_s, d_d = (np.asarray(a, np.uint32) for a in (*ins, *dele))
    return i_s, i_d, _weights(i_s, i_d), d_s, d_d


def _engine(nv, row, col, **cfg):
    w = O.weights(nv, row, col, 1, 0)
    e = sgs.Engine(**cfg)
    e.load_csr(nv, row, col, w)
    return e, Mirror(nv, row, col, w)


# what the snapshot after the failed one does: a deletion that resets one
# vertex, a deletion that resets none, an insert alone, nothing at all
NEXT = {
    "reset": (([], []), ([0], [200])),
    "no reset": (([], []), ([210], [211])),
    "insert": (([201], [202]), ([], [])),
    "empty": (([], []), ([], [])),
}


@pytest.mark.parametrize("nxt", list(NEXT))
@pytest.mark.parametrize("cfg", [dict(), dict(persistent=8), dict(persistent=15), dict(repair=1),
                                 dict(group_size=8), dict(group_size=8, persistent=15)],
                         ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()) or "default")
def test_after_round_limit(cfg, nxt):
    """A path of 100 that one inserted edge connects takes more rounds than the
    limit: the insert reports it, and the next snapshot finishes the path."""
    nv = 300
    a = np.arange(1, 100)
    row, col = O.csr_from_edges(nv, np.concatenate([a, [0, 0, 210]]).astype(np.uint32),
                                np.concatenate([a + 1, [200, 201, 211]]).astype(np.uint32))
    e, m = _engine(nv, row, col, max_rounds=64, **cfg)
    with e:
        qs = e.add_queries([(sgs.SSSP, 0), (sgs.BFS, 0), (sgs.BFS, 200)])
        b = _batch(([0], [1]), ([], []))
        with pytest.raises(sgs.SgsError) as err:
            e.apply_batch(*b)
        assert err.value.code == NOCONV
        m.apply(*b)
        b = _batch(*NEXT[nxt])
        e.apply_batch(*b)
        m.apply(*b)
        for q in qs:
            check_query(q, m, sgs.W_EXPLICIT)
            assert q.stats()["converged"] == 1
        # and from then on as usual
        b = _batch(([50], [250]), ([60], [61]))
        e.apply_batch(*b)
        m.apply(*b)
        for q in qs:
            check_query(q, m, sgs.W_EXPLICIT)


PHASE = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p, C.c_void_p)


class Hooks(C.Structure):
    _fields_ = [("ctx", C.c_void_p), ("before", PHASE), ("after", PHASE)]


def _tree_edges(q, m, n, skip=()):
    par = q.parent()
    v = np.nonzero((par != sgs.INF) & (np.arange(m.nv) != q.source))[0]
    src = np.repeat(np.arange(m.nv), np.diff(m.row).astype(np.int64))
    has = set(zip(src.tolist(), m.col.tolist()))
    out = [(int(par[x]), int(x)) for x in v if (int(par[x]), int(x)) in has and int(x) not in skip]
    return out[::max(1, len(out) // n)][:n]


@pytest.mark.parametrize("phase", ["before", "after"])
@pytest.mark.parametrize("cfg", [dict(), dict(repair=1), dict(group_size=8)],
                         ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()) or "default")
def test_after_user_algorithm_error(cfg, phase):
    nv, row, col = O.rmat_csr(10, 8, 3)
    e, m = _engine(nv, row, col, **cfg)
    with e:
        qs = e.add_queries([(sgs.SSSP, 0), (sgs.BFS, 0), (sgs.CC, 0)])
        fail = PHASE(lambda ctx, g, u: 1)
        ok = PHASE(lambda ctx, g, u: 0)
        hooks = Hooks(None, fail if phase == "before" else ok, fail if phase == "after" else ok)
        app = C.c_int()
        assert sgs.lib().sgs_app_attach(e.h, C.byref(hooks), C.byref(app)) == 0
        edges = _tree_edges(qs[1], m, 40)
        b = _batch(([], []), tuple(zip(*edges)))
        with pytest.raises(sgs.SgsError):
            e.apply_batch(*b)
        if phase == "after":  # the graph update itself has happened
            m.apply(*b)
        assert sgs.lib().sgs_app_detach(e.h, app.value) == 0
        # one more edge, after which little or nothing is reset
        src = np.repeat(np.arange(nv), np.diff(m.row).astype(np.int64))
        dst = int(m.col[-1])
        b = _batch(([], []), ([int(src[-1])], [dst]))
        e.apply_batch(*b)
        m.apply(*b)
        for q in qs:
            check_query(q, m, sgs.W_EXPLICIT)


@pytest.mark.parametrize("cfg", [dict(), dict(group_size=8)],
                         ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()) or "default")
def test_after_pagerank_round_limit(cfg):
    """A PageRank query that cannot reach its tolerance fails every snapshot
    before the integer groups are repaired; once it is gone, the next one is
    exact."""
    nv, row, col = O.rmat_csr(10, 8, 4)
    e, m = _engine(nv, row, col, max_rounds=200, pr_tol=1e-300, **cfg)
    with e:
        qs = e.add_queries([(sgs.SSSP, 0), (sgs.BFS, 0), (sgs.CC, 0)])
        qid = C.c_int()
        assert sgs.lib().sgs_query_add(e.h, sgs.PR, 0, C.byref(qid)) == NOCONV
        b = _batch(([3, 4], [900, 901]), tuple(zip(*_tree_edges(qs[1], m, 30))))
        with pytest.raises(sgs.SgsError) as err:
            e.apply_batch(*b)
        assert err.value.code == NOCONV
        m.apply(*b)
        e.remove_query(qid.value)
        b = _batch(([5], [902]), ([], []))
        e.apply_batch(*b)
        m.apply(*b)
        for q in qs:
            check_query(q, m, sgs.W_EXPLICIT)
