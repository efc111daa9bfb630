"""The exact re-walk's split of a record's free bits (8 thread bits, 5 register bits, the rest
walked; the lowest 7 walked bits through a table) at its edges: no register bits, some, no walked
bits, one, the table full, bits beyond it, and a record split over several CTAs; per-prefix minima
against all energies computed in FP64 on the host, integer Q bit-exact."""
import numpy as np
import pytest

import oracle
import qubo_b200  # noqa: F401
from qubo_b200 import _lib

pytestmark = pytest.mark.gpu


# free bits B = n - A: 1..8 thread bits only, 9..13 register bits, 14 and more walked ones
@pytest.mark.parametrize("n,A", [(3, 2), (9, 1), (10, 1), (13, 1), (14, 1), (15, 1), (16, 3), (20, 0), (21, 1), (22, 9)])
@pytest.mark.parametrize("dtype", [np.int32, np.float64])
def test_prefix_minima_over_the_split(cuda_ok, n, A, dtype):
    rng = np.random.default_rng(100 * n + A)
    Q = (rng.integers(-9, 10, (n, n)) if dtype == np.int32 else rng.standard_normal((n, n))).astype(dtype)
    got = _lib.handle(0).prefix_minima(Q, prefix_bits=A)
    want = oracle.prefix_minima_numpy(Q, A)
    if dtype == np.int32:
        assert np.array_equal(got, want)
    else:  # both sums have at most n^2 additions of values below sum |Q|
        assert np.abs(got - want).max() <= 2 * n * n * 2.0 ** -53 * np.abs(Q).sum()


def _natural(Q, A):
    got = _lib.handle(0).prefix_minima(Q, prefix_bits=A)
    out = np.empty_like(got)
    i = np.arange(1 << A)
    out[i ^ (i >> 1)] = got
    return out


# too many records to be split over CTAs: 7 walked bits (the table full) and 8 (one beyond it),
# against the same minima from records of 4 walked bits
@pytest.mark.parametrize("n", [28, 29])
@pytest.mark.parametrize("dtype", [np.int64, np.float32])
def test_long_walks_agree_with_short_ones(cuda_ok, n, dtype):
    rng = np.random.default_rng(n)
    Q = (rng.integers(-50, 51, (n, n)) if dtype == np.int64 else rng.standard_normal((n, n))).astype(dtype)
    long, short = _natural(Q, 8), _natural(Q, n - 17).reshape(1 << 8, -1).min(axis=1)
    if dtype == np.int64:
        assert np.array_equal(long, short)
    else:
        assert np.abs(long - short).max() <= 2 * n * n * 2.0 ** -53 * np.abs(Q.astype(np.float64)).sum()


def test_many_tied_threads_in_one_record(cuda_ok):
    """Every state of the last variables has the same energy: more tied threads than the CTA's
    winner slots, integer and float (energies from scratch); the smallest key wins."""
    n = 18
    for dtype in (np.int32, np.float64):
        Q = np.zeros((n, n), dtype)
        Q[0, 0], Q[1, 1], Q[0, 1] = -3, -2, 4  # minimum at x0 = 1, x1 = 0, the rest free
        if dtype == np.float64:
            Q *= 0.1
        r = _lib.handle(0).solve(Q)
        ref = oracle.qbf_port(Q)
        assert r["best_X_int"] == ref["best_X_int"] == 1 << (n - 1)
        assert r["best_E"] == Q[0, 0]
