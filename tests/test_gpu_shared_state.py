"""What engines and calls share: launch attributes of a kernel between engines
of different sizes, the buffer that results are gathered through, and a
PageRank job between two updates."""
import threading

import numpy as np
import pytest

import oracle as O
import sgs
from test_gpu_parity import Mirror, check_query

pytestmark = pytest.mark.gpu


def test_engines_of_two_sizes_in_two_threads():
    """Their sweeps ask for different amounts of shared memory."""
    errors = []

    def work(scale):
        try:
            nv, row, col = O.rmat_csr(scale, 8, scale)
            w = O.weights(nv, row, col, 1, 0)
            src = np.repeat(np.arange(nv), np.diff(row).astype(np.int64)).astype(np.uint32)
            with sgs.Engine() as e:
                e.load_csr(nv, row, col, w)
                qs = e.add_queries([(sgs.SSSP, 0), (sgs.BFS, 0), (sgs.CC, 0)])
                for k in range(400):  # the same edges out and in again
                    s = slice(37 * (k // 2), 37 * (k // 2) + 37)
                    none = np.empty(0, np.uint32)
                    if k % 2 == 0:
                        e.apply_batch(none, none, none, src[s], col[s])
                    else:
                        e.apply_batch(src[s], col[s], w[s], none, none)
                m = Mirror(nv, row, col, w)
                for q in qs:
                    check_query(q, m, sgs.W_EXPLICIT)
        except Exception as ex:  # reported by the main thread
            errors.append(ex)

    ts = [threading.Thread(target=work, args=(s,)) for s in (10, 20)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors


def test_gather_gives_memory_back():
    """A large graph's gather keeps no buffer of its size."""
    import torch

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    nv = 1 << 25  # 128 MB of results
    row = np.zeros(nv + 1, np.uint64)
    row[1:] = 1
    with sgs.Engine() as e:
        e.load_csr(nv, row, np.array([1], np.uint32), np.array([3], np.uint32))
        q = e.add_query(sgs.SSSP, 0)
        before = free()
        d = q.value()
        assert d[0] == 0 and d[1] == 3 and np.all(d[2:] == sgs.INF)
        assert before - free() < 64 << 20


def test_pagerank_job_amended_between_long_steps():
    """Updates arrive while a served PageRank job runs: its residual changes
    between two rounds, and the result is the fixed point of the graph it ended on."""
    nv, row, col = O.rmat_csr(13, 16, 8)
    w = O.weights(nv, row, col, 1, 0)
    m = Mirror(nv, row, col, w)
    graphs = [(row, col)]  # by the number of updates applied
    with sgs.Engine() as e:
        e.load_csr(nv, row, col, w)
        i_s, i_d, d_s, d_d = O.gen_updates(nv, row, col, 3, 4000, 4000)
        reqs = [{"kind": "query", "algo": sgs.PR, "value_out": np.empty(nv)}]
        for k in range(8):
            s = slice(500 * k, 500 * k + 500)
            iw = O.weights_pairs(1, i_s[s], i_d[s])
            reqs.append({"kind": "update", "ins_src": i_s[s], "ins_dst": i_d[s], "ins_w": iw,
                         "del_src": d_s[s], "del_dst": d_d[s]})
            m.apply(i_s[s], i_d[s], iw, d_s[s], d_d[s])
            graphs.append((m.row, m.col))
        done = e.serve(reqs, realtime=False)
        assert all(c["status"] == 0 for c in done)
        assert done[0]["version"] >= 2
        ref = O.pagerank(nv, *graphs[done[0]["version"]])
        assert np.max(np.abs(reqs[0]["value_out"] - ref)) <= 1e-6
        q = e.add_query(sgs.SSSP, 0)
        check_query(q, m, sgs.W_EXPLICIT)


def test_served_pagerank_jobs_one_after_the_other():
    """The second job of a trace takes over the first one's vectors; the call
    gives them back."""
    import torch

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    nv = 1 << 22  # 32 MB a vector
    n0, row0, col0 = O.rmat_csr(13, 16, 8)
    row = np.concatenate([row0, np.full(nv - n0, row0[-1], np.uint64)])
    w = O.weights(n0, row0, col0, 1, 0)
    src = np.repeat(np.arange(n0), np.diff(row0).astype(np.int64)).astype(np.uint32)
    m = Mirror(nv, row, col0, w)

    def update(k):  # two of the same size
        d = np.arange(k, len(col0), 97)
        i_s, i_d = np.arange(500 * k, 500 * k + 500, dtype=np.uint32), np.arange(2000, 2500, dtype=np.uint32)
        b = (i_s, i_d, O.weights_pairs(1, i_s, i_d), src[d], col0[d])
        m.apply(*b)
        return dict(zip(("ins_src", "ins_dst", "ins_w", "del_src", "del_dst"), b), kind="update", arrival_s=0.5)

    with sgs.Engine() as e:
        e.load_csr(nv, row, col0, w)
        out = [np.empty(nv) for _ in range(3)]
        pr = [{"kind": "query", "algo": sgs.PR, "arrival_s": 0.4 * k, "value_out": out[k]} for k in range(3)]
        e.serve([pr[0], update(0), pr[2]])  # what an update and a job allocate once
        before = free()
        ref = O.pagerank(nv, m.row, m.col)
        assert np.max(np.abs(out[2] - ref)) <= 1e-6
        done = e.serve([pr[0], pr[1], update(1), pr[2]])
        assert all(c["status"] == 0 for c in done)
        assert before - free() < 16 << 20
        assert done[1]["version"] == 0 and np.max(np.abs(out[1] - ref)) <= 1e-6
        assert done[3]["version"] == 1
        assert np.max(np.abs(out[2] - O.pagerank(nv, m.row, m.col))) <= 1e-6
