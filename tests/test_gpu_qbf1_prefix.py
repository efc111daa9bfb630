"""The int16 QB_F1 tables and search at the edges of the prefix split (8 lower bits whose upper
bits' sums are shared: n = 25 has 7 bits, 26 none above, 27 one above), at the smallest size and
where the grouped walk flips two bits above its groups (n = 31), on wrapping random inputs."""
import numpy as np
import pytest

import oracle
import qubo_b200  # noqa: F401
from conftest import bits_to_int
from qubo_b200.problems import Just_Q
from qubo_b200.solvers import QB_F1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [19, 25, 26, 27, 31])
@pytest.mark.parametrize("amp", [100, 32767])
def test_prefix_edges(cuda_ok, n, amp):
    Q = np.random.default_rng(1000 + n).integers(-amp, amp + 1, (n, n)).astype(np.int16)
    ref = oracle.qbf1_int16_numpy(Q)
    sol = QB_F1().solve(Just_Q(Q), device="cuda", int16_wrap=True)
    assert bits_to_int("".join(map(str, sol.best_X))) == ref["best_X_int"]
    assert sol.best_E == ref["best_E"] and sol.search["exact_E"] == ref["exact_E"]
