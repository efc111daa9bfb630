"""Whole-problem solves with many tied candidate records: split over CTAs while they are few, one CTA
per record when they are many, and the two-phase path when there are more than max_candidates, under
every tie rule against the order of all states."""
import numpy as np
import pytest

import oracle  # noqa: F401
import qubo_b200  # noqa: F401
from qubo_b200 import _lib

pytestmark = pytest.mark.gpu


def _tied(n, step, dtype):
    """Every step-th variable is 1 at the minimum, the others are free: 2^(n - n/step) ties."""
    return (-np.eye(n) * (np.arange(n) % step == 0)).astype(dtype)


def _expected(n, step, rule):
    """The smallest order key among the ties: QBF's inverse-Gray rank of the first n - 20 bits, then
    the rest; natural order; QB_F1's thread, then the rank of the first n - 18 bits, then the suffix."""
    x = np.arange(1 << n, dtype=np.int64)
    must = sum(1 << (n - 1 - i) for i in range(0, n, step))
    x = x[(x & must) == must]

    def rank(g):
        for s in (1, 2, 4, 8, 16):
            g = g ^ (g >> s)
        return g
    if rule == "natural":
        return int(x.min())
    if rule == "qbf":
        B = min(n, 20)
        return int(x[np.lexsort((x & ((1 << B) - 1), rank(x >> B)))[0]])
    s = x & ((1 << 18) - 1)
    tid = ((s >> 10) << 6) | (s & 63)
    p = int((x >> 18)[np.lexsort((rank(x >> 18), tid))[0]])  # the winning prefix, then its smallest suffix
    return int(x[(x >> 18) == p].min())


@pytest.mark.parametrize("n,step", [(20, 3), (22, 2), (24, 6), (24, 2)])
@pytest.mark.parametrize("rule", ["qbf", "natural", "qb_f1"])
@pytest.mark.parametrize("dtype", [np.int32, np.float64])
def test_ties_over_records(cuda_ok, n, step, rule, dtype):
    Q = _tied(n, step, dtype)
    h = _lib.handle(0)
    want, k = _expected(n, step, rule), len(range(0, n, step))
    for form in ("tc", "gray"):
        r = h.solve(Q, form=form, tie_rule=rule)
        assert (r["best_X_int"], r["best_E"]) == (want, -k)
        count = r["candidate_records"]
        for cap in {1, max(1, count - 1), count, count + 1}:
            r = h.solve(Q, form=form, tie_rule=rule, max_candidates=cap)
            assert (r["best_X_int"], r["best_E"], r["candidate_records"]) == (want, -k, count)
