"""The segmented map (csrc/sgs_segmap.cuh, a public header of user algorithms)
over frontiers of any lengths: every slot of every entry is visited once, also
beside entries without slots."""
import ctypes as C
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    L = C.CDLL(os.path.join(REPO, "c-gpustreamgraph_b200", "lib", "libsgs_segmap_test.so"))
    L.sgs_test_segmap.argtypes = [C.c_uint32, C.c_void_p, C.c_int, C.c_uint32, C.c_void_p, C.c_void_p]
    return L


def _lengths(kind):
    rng = np.random.default_rng(len(kind))
    return {
        "no zeros": rng.integers(1, 40, 3000),
        "ones": np.ones(3000),
        "some zeros": np.where(rng.random(3000) < 0.2, 0, rng.integers(1, 40, 3000)),
        "mostly zeros": np.where(rng.random(5000) < 0.95, 0, rng.integers(1, 9, 5000)),
        "zeros between large ones": np.tile([0, 0, 3000, 0, 5, 1500, 0], 12),
        "zeros at the chunk's edge": np.concatenate([np.full(250, 3), np.zeros(12), np.full(250, 5), np.zeros(1)]),
        "a chunk of zeros": np.concatenate([[7], np.zeros(600), [9, 0, 4]]),
        "zeros first and last": np.concatenate([np.zeros(40), np.arange(1, 90), np.zeros(300)]),
        "nothing but zeros": np.zeros(500),
    }[kind].astype(np.uint32)


@pytest.mark.parametrize("ctas", [1, 7, 300])
@pytest.mark.parametrize("quad", [0, 1])
@pytest.mark.parametrize("kind", ["no zeros", "ones", "some zeros", "mostly zeros", "zeros between large ones",
                                  "zeros at the chunk's edge", "a chunk of zeros", "zeros first and last",
                                  "nothing but zeros"])
def test_every_slot_once(lib, kind, quad, ctas):
    n = _lengths(kind)
    total = int(n.sum())
    seen = np.zeros(max(total, 1), np.uint32)
    counted = np.zeros(1, np.uint64)
    assert lib.sgs_test_segmap(len(n), n.ctypes.data, quad, ctas, seen.ctypes.data, counted.ctypes.data) == 0
    assert np.all(seen[:total] == 1)
    assert counted[0] == total
