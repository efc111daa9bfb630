"""The 16-bit pair kernel's low t bits (variables n-17 .. n-19: K slots of the MMA, two digits
per coupling row) at the edges of their range: rows far beyond one digit's 2048, both signs,
with the pair variable n-16 coupled as strongly, at the smallest sizes (two blocks of 16 tiles
at n = 20) and with shards that start inside a 32-block run of the block walk."""
import numpy as np
import pytest

import oracle
import qubo_b200  # noqa: F401
from qubo_b200 import _lib

pytestmark = pytest.mark.gpu


def _wide_rows(n, seed):
    """Integer Q, sum |Q| <= 2^22, whose low t rows span most of the 16-bit value range."""
    rng = np.random.default_rng(seed)
    Q = np.triu(rng.integers(-30, 31, (n, n)))
    Q[n - 17, n - 1], Q[n - 17, n - 8] = 9000, -14000
    Q[n - 18, n - 5], Q[n - 18, n - 2] = -2049, 2048
    Q[n - 19, n - 7] = -13000
    Q[n - 16, n - 4], Q[n - 16, n - 6] = 6000, -7000  # a half position and a chunk bit of the pair's row
    return Q.astype(np.int32)


@pytest.mark.parametrize("n", [20, 21, 23, 26])
@pytest.mark.parametrize("sign", [1, -1])
def test_low_t_rows_of_both_digits(cuda_ok, n, sign):
    Q = sign * _wide_rows(n, n)
    ref = oracle.qbf_port(Q)
    h = _lib.handle(0)
    r = h.solve(Q, form="tc")
    assert r["plan"]["tc_kernel"] == "pair_u16" and r["err_bound"] == 0.0
    assert (r["best_X_int"], r["best_E_int"]) == (ref["best_X_int"], ref["best_E"])
    assert r["pass1_min"] == ref["best_E"]
    b = h.solve_batch([Q, _wide_rows(24, 1), Q])
    assert [x["best_X_int"] for x in b[::2]] == [ref["best_X_int"]] * 2
    mins = []
    for s in range(7):  # seven shards: uneven runs of record blocks
        mins.append(h.solve_begin(Q, form="tc", shard_index=s, shard_count=7))
        h.solve_finish(mins[-1], n)
    assert min(mins) == ref["best_E"]
