"""Performance cases of the streaming-graph engine.

Each case is one kind of work that a program using this framework repeats,
called through the public entry points:

* ``snapshot``  -- a snapshot of edge inserts and deletes applied to a graph
  that keeps SSSP, BFS and CC queries up to date, then the queries' values
  read back (the engine's main path);
* ``pagerank``  -- the same for a PageRank query;
* ``batched``   -- the same for many BFS/SSSP sources at once (wide groups);
* ``query``     -- queries added to a loaded graph, converged from scratch,
  read back and removed;
* ``serve``     -- a closed-loop trace of updates and one-shot queries;
* ``ppr``       -- differentiable personalized PageRank, forward and backward.

Graphs are R-MAT (0.57/0.19/0.19/0.05, duplicates and self-loops removed)
with any number of vertices; weights are uniform in [1, 64].  The update
stream is a ring of disjoint edge sets, half of each set edges of the graph
and half uniform new pairs: pass k inserts set k and deletes set k + 1, so
every set is deleted and comes back some snapshots later and the graph's size
stays the same however many passes are run.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "c-gpustreamgraph_b200"))

import sgs  # noqa: E402
from sgs.autograd import personalized_pagerank  # noqa: E402

ALPHA = 0.85
RING = 4  # edge sets of the update ring


def listed():
    return [
        # a small graph with a few updates at a time, numpy in and out: what
        # an interactive user or a test does; launches and host reads count
        dict(name="snapshot_small", kind="snapshot", nv=1000, ef=12, updates=75, mem="host", budget=0.0),
        # an ordinary snapshot on a graph that sits in L2 (the command line
        # tools' sizes), numpy in and out
        dict(name="snapshot_s16", kind="snapshot", nv=65536, ef=16, updates=10000, mem="host", budget=0.0),
        # an ordinary snapshot on a graph larger than L2, device arrays; odd sizes
        dict(name="snapshot_1m", kind="snapshot", nv=1000003, ef=16, updates=99999, mem="device", budget=0.0),
        # the largest: scale 24, a million updates per snapshot
        dict(name="snapshot_s24", kind="snapshot", nv=1 << 24, ef=16, updates=500000, mem="device", budget=0.0),
        # most of the graph in pinned host memory behind the edge cache
        dict(name="snapshot_host", kind="snapshot", nv=1 << 20, ef=16, updates=50000, mem="device", budget=0.35),
        # incremental PageRank, 10,000 inserts and deletes at scale 16
        dict(name="pagerank_s16", kind="pagerank", nv=65536, ef=16, updates=10000),
        # incremental PageRank on a graph whose in-edges exceed L2
        dict(name="pagerank_2m", kind="pagerank", nv=2000000, ef=16, updates=250000),
        # a full wide group of BFS and SSSP sources through a snapshot
        dict(name="batched_64", kind="batched", nv=1 << 18, ef=16, lanes=64, updates=25000),
        # one-shot SSSP and BFS queries on a loaded graph, results on the host
        dict(name="query_1m", kind="query", nv=1 << 20, ef=16, algos="sssp,bfs", pull=1),
        # a served trace: updates among one-shot queries
        dict(name="serve_s16", kind="serve", nv=65536, ef=16, updates=1000, queries=24, width=4),
        # PPR training step, small graph and few teleport vectors
        dict(name="ppr_small", kind="ppr", nv=4096, ef=16, K=8, dtype="f64"),
        # PPR training step, 64 teleport vectors on a million vertices
        dict(name="ppr_1m", kind="ppr", nv=1 << 20, ef=16, K=64, dtype="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["snapshot", "snapshot", "snapshot", "pagerank", "batched", "query", "serve", "ppr", "ppr"])
    ef = rng.randint(8, 20)
    if kind == "snapshot":
        mem = rng.choice(["host", "device"])
        budget = rng.choice([0.0, 0.0, 0.0, round(rng.uniform(0.2, 0.8), 2)])
        nv = _log(rng, 900, 1 << 20 if mem == "host" or budget else 1 << 23)
        return dict(kind=kind, nv=nv, ef=ef, updates=max(8, _log(rng, nv * 0.005, nv * 0.1)), mem=mem, budget=budget)
    if kind == "pagerank":
        nv = _log(rng, 3000, 2000000)
        return dict(kind=kind, nv=nv, ef=ef, updates=max(8, _log(rng, nv * 0.005, nv * 0.15)))
    if kind == "batched":
        nv = _log(rng, 3000, 1 << 18)
        return dict(kind=kind, nv=nv, ef=ef, lanes=rng.randint(5, 100), updates=max(8, _log(rng, nv * 0.005, nv * 0.1)))
    if kind == "query":
        algos = rng.choice(["sssp", "bfs", "cc", "sssp,bfs", "bfs,cc", "sssp,bfs,cc,sssp"])
        return dict(kind=kind, nv=_log(rng, 900, 1 << 21), ef=ef, algos=algos, pull=rng.choice([1, 3]))
    if kind == "serve":
        nv = _log(rng, 3000, 1 << 18)
        return dict(kind=kind, nv=nv, ef=ef, updates=max(8, _log(rng, nv * 0.002, nv * 0.03)),
                    queries=rng.randint(8, 40), width=rng.choice([4, 16, 64]))
    nv = _log(rng, 900, 1 << 19)
    return dict(kind=kind, nv=nv, ef=ef, K=_log(rng, 1, 64), dtype=rng.choice(["f64", "f32"]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _graph(nv, ef, gen):
    """nv * ef R-MAT edges among nv vertices: sorted unique keys (src << 32 | dst)."""
    scale, ne = max(1, (nv - 1).bit_length()), nv * ef
    key = torch.empty(0, dtype=torch.int64, device="cuda")
    while key.numel() < ne:
        m = ne + ne // 4
        u = torch.zeros(m, dtype=torch.int32, device="cuda")
        v = torch.zeros(m, dtype=torch.int32, device="cuda")
        for _ in range(scale):
            r = torch.rand(m, generator=gen, device="cuda")
            u.mul_(2).add_(r >= 0.76)
            v.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        ok = (u != v) & (u < nv) & (v < nv)
        key = torch.unique(torch.cat([key, (u[ok].to(torch.int64) << 32) | v[ok].to(torch.int64)]))
    drop = key.numel() - ne
    if drop:
        keep = torch.ones(key.numel(), dtype=torch.bool, device="cuda")
        keep[_pick(key.numel(), drop, gen)] = False
        key = key[keep]
    return key


def _csr(key, nv):
    """Row offsets (int64) and columns (int32) of sorted keys."""
    row = torch.searchsorted(key, torch.arange(nv + 1, dtype=torch.int64, device="cuda") << 32)
    return row, (key & 0xFFFFFFFF).to(torch.int32)


def _weights(n, gen):
    return torch.randint(1, 65, (n,), generator=gen, device="cuda", dtype=torch.int32)


def _pick(n, k, gen):
    """k distinct indices below n, in random order."""
    i = torch.unique(torch.randint(0, n, (k + k // 8 + 64,), generator=gen, device="cuda"))
    while i.numel() < k:
        i = torch.unique(torch.cat([i, torch.randint(0, n, (k + 64,), generator=gen, device="cuda")]))
    return i[torch.randperm(i.numel(), generator=gen, device="cuda")][:k]


def _new_pairs(key, nv, k, gen):
    """Keys of k distinct uniform pairs that are no edges, in random order."""
    got = key.new_empty(0)
    while got.numel() < k:
        c = 2 * k + 64
        u = torch.randint(0, nv, (c,), generator=gen, device="cuda")
        v = torch.randint(0, nv, (c,), generator=gen, device="cuda")
        p = ((u << 32) | v)[u != v]
        at = torch.searchsorted(key, p).clamp_(max=key.numel() - 1)
        got = torch.unique(torch.cat([got, p[key[at] != p]]))
    return got[torch.randperm(got.numel(), generator=gen, device="cuda")][:k]


def _stream(case, seed):
    """The graph without the ring's set 0, and the ring's sets (keys, weights)."""
    gen = _gen(seed)
    nv, n = case["nv"], case["updates"]
    key = _graph(nv, case["ef"], gen)
    n = min(n, key.numel() // (4 * RING))
    old = n // 2
    new = _new_pairs(key, nv, RING * (n - old), gen).reshape(RING, -1)
    idx = _pick(key.numel(), RING * old, gen).reshape(RING, -1)
    sets = []
    for j in range(RING):
        s = torch.cat([key[idx[j]], new[j]])
        s = s[torch.randperm(n, generator=gen, device="cuda")]
        sets.append((s, _weights(n, gen)))
    keep = torch.ones(key.numel(), dtype=torch.bool, device="cuda")
    keep[idx.reshape(-1)] = False
    # edges outside the ring, then sets 1.. with their own weights
    base = key[keep]
    allk = torch.cat([base] + [s for s, _ in sets[1:]])
    allw = torch.cat([_weights(base.numel(), gen)] + [w for _, w in sets[1:]])
    allk, order = torch.sort(allk)
    return allk, allw[order], sets, gen


def _ck(rc):
    if rc != sgs.OK:
        raise sgs.SgsError(rc, sgs.lib().sgs_last_error().decode())


def _load(engine, nv, key, w):
    row, col = _csr(key, nv)
    torch.cuda.synchronize()
    _ck(sgs.lib().sgs_load_csr(engine.h, nv, row.data_ptr(), col.data_ptr(), w.data_ptr(), sgs.MEM_DEVICE))
    engine.nv = nv


def _split(s, host):
    k, w = s
    parts = [(k >> 32).to(torch.int32), (k & 0xFFFFFFFF).to(torch.int32), w]
    return [p.cpu().numpy().view(np.uint32) for p in parts] if host else parts


def _sources(key, count, gen):
    """Vertices with out-edges, uniformly."""
    v = torch.unique_consecutive(key >> 32)
    return [int(x) for x in v[torch.randint(0, v.numel(), (count,), generator=gen, device="cuda")]]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ppr":
        return _prepare_ppr(case, seed)
    nv = case["nv"]
    if kind == "query":
        gen = _gen(seed)
        key = _graph(nv, case["ef"], gen)
        e = sgs.Engine(pull=case["pull"])
        _load(e, nv, key, _weights(key.numel(), gen))
        algos = case["algos"].split(",")
        src = _sources(key, 8 * len(algos), gen)
        specs = [[(a, src[i * len(algos) + j]) for j, a in enumerate(algos)] for i in range(8)]
        return dict(case=case, e=e, specs=specs, k=0)
    key, w, sets, gen = _stream(case, seed)
    cfg = {}
    if kind == "snapshot" and case["budget"]:
        gb = key.numel() * 8 / 1e9
        cfg = dict(hbm_budget_gb=case["budget"] * gb, cache_gb=0.3 * case["budget"] * gb)
    if kind == "batched":
        cfg = dict(group_size=64)
    if kind == "serve":
        # every query sees exactly the updates before it
        cfg = dict(group_size=case["width"], serve_restarts=0)
    e = sgs.Engine(**cfg)
    _load(e, nv, key, w)
    host = kind in ("pagerank", "serve") or case.get("mem") == "host"
    st = dict(case=case, e=e, sets=[_split(s, host) for s in sets], k=0, host=host)
    if kind == "snapshot":
        st["q"] = e.add_queries([(sgs.SSSP, 0), (sgs.BFS, 0), (sgs.CC, 0)])
    elif kind == "pagerank":
        st["q"] = [e.add_query(sgs.PR)]
    elif kind == "batched":
        src = _sources(key, case["lanes"], gen)
        st["q"] = e.add_queries([(sgs.SSSP if i % 2 else sgs.BFS, s) for i, s in enumerate(src)])
    else:
        st["src"] = _sources(key, case["queries"], gen)
    if kind != "serve" and not host:
        st["out"] = torch.empty((len(st["q"]), nv), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return st


def _ppr_inputs(case, seed):
    gen = _gen(seed)
    nv, K = case["nv"], case["K"]
    row, col = _csr(_graph(nv, case["ef"], gen), nv)
    dt = torch.float64 if case["dtype"] == "f64" else torch.float32
    # weights log-uniform in [0.1, 10], teleport vectors uniform over 32 seeds
    w = torch.exp((torch.rand(col.numel(), generator=gen, device="cuda", dtype=torch.float64) - 0.5)
                  * (2 * math.log(10.0))).to(dt)
    T = torch.zeros((nv, K), dtype=dt, device="cuda")
    T.scatter_(0, torch.randint(0, nv, (32, K), generator=gen, device="cuda"), 1.0 / 32)
    return row, col, w, T, _pick(nv, min(1024, nv // 2), gen)


def _prepare_ppr(case, seed):
    row, col, w, T, target = _ppr_inputs(case, seed)
    graph = sgs.Ppr(case["nv"], row.cpu().numpy().view(np.uint64), col.cpu().numpy().view(np.uint32))
    return dict(case=case, graph=graph, w=w.requires_grad_(), T=T.requires_grad_(), target=target)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _apply(st):
    e, k = st["e"], st["k"]
    ins, dele = st["sets"][k % RING], st["sets"][(k + 1) % RING]
    st["k"] = k + 1
    if st["host"]:
        e.apply_batch(ins[0], ins[1], ins[2], dele[0], dele[1])
    else:
        e.apply_batch_ptr(ins[0].data_ptr(), ins[1].data_ptr(), ins[2].data_ptr(), len(ins[0]),
                          dele[0].data_ptr(), dele[1].data_ptr(), len(dele[0]), sgs.MEM_DEVICE)


def _signed(a):
    """uint32 values as int32 (a view)."""
    return a.view(np.int32) if a.dtype == np.uint32 else a


def run(st):
    kind = st["case"]["kind"]
    if kind == "ppr":
        w, T = st["w"], st["T"]
        w.grad = T.grad = None
        # the tolerance of the gradient checks: at the default one a large
        # graph's scores end 3e-8 short of the fixed point, so two runs could
        # only be compared by where they stopped
        X = personalized_pagerank(st["graph"], w, T, alpha=ALPHA, tol=1e-16 * T.numel())
        X[st["target"]].sum().backward()
        return dict(X=X.detach(), dw=w.grad, dT=T.grad)
    e = st["e"]
    if kind == "query":
        k = st["k"]
        st["k"] = k + 1
        qs = e.add_queries(st["specs"][k % len(st["specs"])])
        out = [_signed(q.value()) for q in qs]
        for q in qs:
            e.remove_query(q)
        return out
    if kind == "serve":
        return _run_serve(st)
    _apply(st)
    if st["host"]:
        return [_signed(q.value()) for q in st["q"]]
    out = st["out"]
    for i, q in enumerate(st["q"]):
        _ck(sgs.lib().sgs_gather(e.h, q.qid, sgs.FIELD_VALUE, out[i].data_ptr(), sgs.MEM_DEVICE))
    return out


def _run_serve(st):
    """The ring's sets as updates (one turn of the ring, so the graph ends as
    it began) spread over the queries."""
    src, nq = st["src"], len(st["src"])
    out = np.empty((nq, st["e"].nv), np.uint32)
    trace, done = [], 0
    for i, s in enumerate(src):
        while done < RING and done * nq <= i * RING:
            ins, dele = st["sets"][done], st["sets"][(done + 1) % RING]
            trace.append(dict(kind="update", ins_src=ins[0], ins_dst=ins[1], ins_w=ins[2],
                              del_src=dele[0], del_dst=dele[1]))
            done += 1
        trace.append(dict(kind="query", algo=sgs.SSSP if i % 2 else sgs.BFS, source=s, value_out=out[i]))
    res = st["e"].serve(trace, realtime=False)
    if any(r["status"] != sgs.OK for r in res):
        raise RuntimeError("a served request failed")
    return _signed(out)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    nv, kind = case["nv"], case["kind"]
    ne = nv * case["ef"]
    # a snapshot: the batch read (ids, weights), the changed slots written
    upd = case.get("updates", 0) * (12 + 8 + 8 + 4)
    if kind == "snapshot":  # and three value vectors
        return dict(bytes=upd + 3 * 4 * nv, flops=0)
    if kind == "batched":
        return dict(bytes=upd + 4 * nv * case["lanes"], flops=0)
    if kind == "pagerank":  # one pass over the in-edges and the vector
        return dict(bytes=upd + 4 * ne + 24 * nv, flops=2 * ne)
    if kind == "query":  # the graph once (weights for SSSP) and the values
        a = case["algos"].split(",")
        return dict(bytes=ne * (8 if "sssp" in a else 4) + 4 * nv * len(a), flops=0)
    if kind == "serve":
        return dict(bytes=RING * upd + case["queries"] * (8 * ne / 4 + 4 * nv), flops=0)
    s = 8 if case["dtype"] == "f64" else 4
    K = case["K"]
    # one step each way and the edge gradient: ids and weights, T in, X, dT
    # and dw out; a multiply-add per edge and column each
    return dict(bytes=ne * (4 + 2 * s) + nv * K * (2 * s + 8), flops=6 * ne * K)


# ---------------------------------------------------------------------------
# the same values in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "pagerank":
        return _exact_pagerank(case, seed)
    if case["kind"] == "ppr":
        return _exact_ppr(case, seed)
    return None  # integers


def _exact_pagerank(case, seed):
    nv = case["nv"]
    key, _, sets, _ = _stream(case, seed)
    drop = torch.sort(sets[1][0]).values
    at = torch.searchsorted(drop, key).clamp_(max=drop.numel() - 1)
    key = torch.cat([key[drop[at] != key], sets[0][0]])
    src, dst = key >> 32, key & 0xFFFFFFFF
    deg = torch.bincount(src, minlength=nv).double()
    inv = torch.where(deg > 0, ALPHA / deg.clamp(min=1), torch.zeros_like(deg))
    x = torch.full((nv,), 1 - ALPHA, dtype=torch.float64, device="cuda")
    for _ in range(400):
        y = torch.full_like(x, 1 - ALPHA).index_add_(0, dst, (x * inv)[src])
        change = float((y - x).abs().sum())
        x = y
        if change < 1e-12 * nv:
            break
    return [x.cpu().numpy()]


def _exact_ppr(case, seed):
    row, col, w, T, target = _ppr_inputs(case, seed)
    nv, K = case["nv"], case["K"]
    w, T = w.double(), T.double()
    src = torch.repeat_interleave(torch.arange(nv, device="cuda"), row[1:] - row[:-1])
    s = torch.zeros(nv, dtype=torch.float64, device="cuda").index_add_(0, src, w)
    p = w / s[src]
    P = torch.sparse_csr_tensor(row, col.to(torch.int64), p, (nv, nv))
    order = torch.argsort(col, stable=True)
    crow = torch.searchsorted(col[order].to(torch.int64), torch.arange(nv + 1, device="cuda"))
    PT = torch.sparse_csr_tensor(crow, src[order], p[order], (nv, nv))

    def fixed(A, b):
        x = b.clone()
        for _ in range(400):
            y = b + ALPHA * (A @ x)
            change = float((y - x).abs().sum())
            x = y
            if change < 1e-18 * nv * K:
                break
        return x

    X = fixed(PT, (1 - ALPHA) * T)
    G = torch.zeros((nv, K), dtype=torch.float64, device="cuda")
    G[target] = 1.0
    Y = fixed(P, G)
    c = (X * (G - Y)).sum(1)
    dw = torch.empty_like(w)
    step = max(1, (1 << 28) // K)
    for i in range(0, w.numel(), step):
        u, v = src[i:i + step], col[i:i + step].to(torch.int64)
        dw[i:i + step] = (ALPHA * (X[u] * Y[v]).sum(1) + c[u]) / s[u]
    return dict(X=X, dw=dw, dT=(1 - ALPHA) * Y)

