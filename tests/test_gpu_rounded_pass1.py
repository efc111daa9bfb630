"""Pass-1 values of the 16-bit pair form off the exact path (matrices rounded to integers in units
of 1/sigma): how far the smallest one may lie from the FP64 minimum."""
import numpy as np
import pytest

import qubo_b200  # noqa: F401
from qubo_b200 import _lib

pytestmark = pytest.mark.gpu

PAIR16 = _lib.TC_KERNELS[4]


# float Q, and integer Q beyond 2^22; the couplings of the low t bits (variables n-17 .. n-19) with the
# last eight variables five times as wide as the rest
@pytest.mark.parametrize("n", [20, 21, 23, 26])
@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.int64])
def test_error_bound_holds(cuda_ok, n, dtype):
    for seed in range(8):
        rng = np.random.default_rng([n, seed])
        Q = rng.uniform(-1, 1, (n, n))
        Q[n - 19:n - 16, n - 8:] *= 5
        Q = (Q * (1 << 30)).astype(dtype) if dtype == np.int64 else Q.astype(dtype)
        r = _lib.handle(0).solve(Q, form="tc")
        assert r["plan"]["tc_kernel"] == PAIR16 and r["err_bound"] > 0
        assert abs(r["pass1_min"] - r["best_E"]) <= r["err_bound"]


@pytest.mark.parametrize("n", [20, 24])
@pytest.mark.parametrize("sign", [1, -1])
def test_ten_rows_rounded_the_same_way(cuda_ok, n, sign):
    """The minimum's seven y rows, three low t rows and column energy all lose 0.49 units to the
    same side.  With the t variables' sum rounded as one value that is 4.5 units at most (seven
    rows, the sum, the column energy); each row by itself would lose 5.39."""
    f = 0.49 * sign
    Q = np.zeros((n, n))
    i = np.arange(n)
    Q[i, i] = 100.0
    y, low, u = n - 9 - np.arange(7), n - 17 - np.arange(3), n - 1
    Q[y, y] = Q[low, low] = -50.0
    Q[y, u] = -200.0 - f
    Q[low, u] = -300.0 - f
    Q[u, u] = -1000.0 - f
    Q[n - 2, n - 2] = 36000.0  # the span that makes the unit 1
    r = _lib.handle(0).solve(Q, form="tc")
    S = np.abs(Q).sum()
    assert r["plan"]["tc_kernel"] == PAIR16 and abs(10.0 / (r["err_bound"] - S * 2.0 ** -16) - 1.0) < 1e-9
    assert r["best_X_int"] == sum(1 << (n - 1 - v) for v in [*y, *low, u])
    assert abs(r["pass1_min"] - r["best_E"]) <= 4.5 + S * 2.0 ** -18
