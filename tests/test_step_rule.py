"""The arithmetic of PPR's step lengths on the CPU: sums of terms rounded to
2^-47 of a norm come out the same in any order and are off by no more than the
slack that the end of the iteration adds; the helper that the GPU tests place
their limits with finds the long step that removes a Perron vector."""
import numpy as np
import pytest

import step_rule as S


def _unit(norm):
    return 2.0 ** np.floor(np.log2(norm))


@pytest.mark.parametrize("growth", [1e-9, 0.3, 0.85, 1.0, 7.9])
@pytest.mark.parametrize("scale", [1e-12, 1.0, 3e7])
def test_exact_sums(growth, scale):
    rng = np.random.default_rng(int(1e3 * growth))
    n = 20000
    x = rng.random(n) ** 8
    x *= growth * scale / x.sum()  # the norm before is `scale`
    unit = _unit(scale)
    c = 48.0 * unit
    terms = (x + c) - c
    sums = set()
    for _ in range(20):
        p = rng.permutation(n)
        acc = 0.0
        for part in np.array_split(terms[p], rng.integers(1, 40)):
            s = 0.0
            for t in part:
                s += t
            acc += s
        sums.add(acc)
    assert len(sums) == 1
    slack = n * (unit * 2.0**-48)
    # (the reference sum is correctly rounded)
    import math

    assert abs(sums.pop() - math.fsum(x)) <= slack


def test_first_long_step_removes_the_perron_vector():
    rng = np.random.default_rng(1)
    n, alpha = 60, 0.85
    P = rng.random((n, n))
    P /= P.sum(1, keepdims=True)
    T = np.zeros((n, 1))
    T[3] = 1.0
    k, norms = S.first_long_step(P.T, 1 - alpha, T, alpha)
    assert k is not None and 3 <= k < 10
    ratio = norms[-1] / norms[-2]
    assert abs(ratio - alpha) < 1e-2  # column sums of alpha P^T
