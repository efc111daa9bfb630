"""The int16 QB_F1 search reports groups of 32 steps and the exact step is found afterwards: inputs
full of ties (the earliest step, the lowest thread and the first suffix win) and inputs whose
minima wrap, at the largest size of the per-step walk (n = 28: 16 steps per chunk), the smallest
of the grouped one (n = 29: one group per chunk) and the first with two groups per chunk."""
import numpy as np
import pytest

import oracle
import qubo_b200  # noqa: F401
from conftest import bits_to_int
from qubo_b200.problems import Just_Q
from qubo_b200.solvers import QB_F1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [28, 29, 30])
@pytest.mark.parametrize("kind", ["ties", "zero", "wrap"])
def test_groups(cuda_ok, n, kind):
    rng = np.random.default_rng(n)
    if kind == "ties":  # few couplings of one size: many states of minimal energy
        Q = np.triu(rng.integers(-1, 2, (n, n)) * (rng.random((n, n)) < 0.15))
    elif kind == "zero":
        Q = np.zeros((n, n))
    else:
        Q = rng.integers(-32768, 32768, (n, n))
    Q = Q.astype(np.int16)
    ref = oracle.qbf1_int16_numpy(Q)
    sol = QB_F1().solve(Just_Q(Q), device="cuda", int16_wrap=True)
    assert bits_to_int("".join(map(str, sol.best_X))) == ref["best_X_int"]
    assert sol.best_E == ref["best_E"] and sol.search["exact_E"] == ref["exact_E"]
