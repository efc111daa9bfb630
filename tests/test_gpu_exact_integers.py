"""Integer Q with energies beyond 2^52, where FP64 holds whole numbers but no halves: every
reported energy is the exact integer (sum |Q| < 2^53), against all energies in int64."""
import numpy as np
import pytest

import qubo_b200  # noqa: F401
from qubo_b200 import _lib

pytestmark = pytest.mark.gpu


def _energies(Q):
    n = Q.shape[0]
    X = (np.arange(1 << n)[:, None] >> np.arange(n - 1, -1, -1)) & 1
    return ((X @ Q) * X).sum(axis=1)


def _heavy(n, seed):
    """One diagonal entry of -1.5 * 2^52 and odd couplings beside it."""
    rng = np.random.default_rng(seed)
    Q = np.triu(2 * rng.integers(-500, 500, (n, n)) + 1).astype(np.int64)
    Q[0, 0] = -3 * 2 ** 51
    return Q


def test_one_odd_coupling_beside_2_to_52(cuda_ok):
    Q = np.zeros((16, 16), np.int64)
    Q[0, 0], Q[0, 1] = -2 ** 52, -1
    got = _lib.handle(0).prefix_minima(Q, prefix_bits=2)  # prefixes 00, 01, 11, 10
    assert [int(v) for v in got] == [0, 0, -2 ** 52 - 1, -2 ** 52]


# free bits n - A: thread bits alone, register bits, walked bits
@pytest.mark.parametrize("n,A", [(12, 4), (16, 4), (18, 3)])
def test_prefix_minima(cuda_ok, n, A):
    Q = _heavy(n, n)
    got = _lib.handle(0).prefix_minima(Q, prefix_bits=A)
    i = np.arange(1 << A)
    want = _energies(Q).reshape(1 << A, -1).min(axis=1)[i ^ (i >> 1)]
    assert [int(v) for v in got] == [int(v) for v in want]


@pytest.mark.parametrize("n,form,rule", [(16, "exact", "qbf"), (16, "exact", "natural")] +
                         [(20, form, rule) for form in ("exact", "gray", "tc") for rule in ("qbf", "natural", "qb_f1")])
def test_solve(cuda_ok, n, form, rule):
    Q = _heavy(n, n + 1)
    E = _energies(Q)
    assert (E == E.min()).sum() == 1 and np.abs(Q).sum() < 2 ** 53
    r = _lib.handle(0).solve(Q, form=form, tie_rule=rule)
    assert (r["best_X_int"], r["best_E_int"]) == (int(E.argmin()), int(E.min()))
