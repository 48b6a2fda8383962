"""Which first round the repair of a narrow group takes, seen in the sweep's
own counts: the restricted one reads 4 bytes per slot walked, the full one 8
with explicit weights and relaxes every (lane, edge) pair it walks.  All
weight modes, against the oracle."""
import numpy as np
import pytest

import oracle as O
import sgs
from test_gpu_parity import Mirror, check_query

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wmode", [sgs.W_EXPLICIT, sgs.W_SYNTH, sgs.W_UNIT])
@pytest.mark.parametrize("scale", [12, 16])
def test_repair_mode_taken(scale, wmode):
    nv, row, col = O.rmat_csr(scale, 16, 6)
    ew = wmode == sgs.W_EXPLICIT
    w = O.weights(nv, row, col, 1, 0) if ew else None
    rng = np.random.default_rng(scale)
    with sgs.Engine(weight_mode=wmode) as e:
        e.load_csr(nv, row, col, w)
        m = Mirror(nv, row, col, w if ew else np.ones(len(col), np.uint32))
        qs = e.add_queries([(sgs.SSSP, 0), (sgs.BFS, 0), (sgs.CC, 0), (sgs.SSSP, 5)])
        e.kernel_timing(True)

        def step(n_del):
            src = np.repeat(np.arange(nv), np.diff(m.row).astype(np.int64)).astype(np.uint32)
            k = rng.choice(len(m.col), n_del, replace=False)
            i_s, i_d = rng.integers(0, nv, (2, 200)).astype(np.uint32)
            keep = i_s != i_d
            i_s, i_d = i_s[keep], i_d[keep]
            i_w = O.weights_pairs(1, i_s, i_d) if ew else np.ones(len(i_s), np.uint32)
            e.kernel_timing(True)
            e.apply_batch(i_s, i_d, i_w if ew else None, src[k], m.col[k])
            m.apply(i_s, i_d, i_w, src[k], m.col[k])
            for q in qs:
                check_query(q, m, wmode)
            resets = sum(q.stats()["invalidated"] for q in qs)
            return resets, e.kernel_stats()["group_sweep"]

        # a few deletions: restricted; the walk tests every slot and relaxes
        # few pairs, so 8 bytes for each of those are far below 4 a slot
        resets, k = step(nv // 16)
        assert 0 < resets <= nv // 2
        assert k["launches"] == 1 and k["slots"] > 0
        pairs = (k["bytes_alg"] - 4 * k["slots"] - 20 * k["entries"]) / 8
        assert 0 <= pairs < 0.5 * k["slots"]
        # a third of the edges: full; a vertex walked is reached in a lane at
        # least, so its live edges are pairs (slots are padded to four per
        # vertex, and a block keeps tombstones below a sixteenth of its edges)
        resets, k = step(len(m.col) // 3)
        assert resets > nv // 2
        per_slot = 8 if ew else 4
        pairs = (k["bytes_alg"] - per_slot * k["slots"] - 20 * k["entries"]) / 8
        assert k["launches"] == 1 and pairs * 17 / 16 + 3 * k["entries"] >= k["slots"]
