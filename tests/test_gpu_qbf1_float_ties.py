"""QB_F1's order on float matrices of tenths, whose many tied states differ by rounding alone: whole
and sharded searches answer with a minimal state and its energy."""
import numpy as np
import pytest

import oracle  # noqa: F401
import qubo_b200  # noqa: F401
from qubo_b200 import _lib

pytestmark = pytest.mark.gpu


def _sharded(h, Q, form, shards):
    n = Q.shape[0]
    opts = dict(form=form, tie_rule="qb_f1", shard_count=shards)
    lowest = min(h.solve_begin(Q, shard_index=s, **opts) for s in range(shards))
    out = []
    for s in range(shards):
        h.solve_begin(Q, shard_index=s, **opts)
        out.append(h.solve_finish(lowest, n))
    return min((r for r in out if r["found"]), key=lambda r: r["best_E"])


@pytest.mark.parametrize("n", [19, 20, 21])
@pytest.mark.parametrize("form", ["exact", "auto"])
def test_ties_to_within_rounding(cuda_ok, n, form):
    h = _lib.handle(0)
    X = ((np.arange(1 << n)[:, None] >> np.arange(n - 1, -1, -1)) & 1).astype(np.int64)
    for seed in range(12):
        T = np.random.default_rng([seed, n]).integers(-3, 4, (n, n))
        lowest = int(((X @ T) * X).sum(axis=1).min())  # in tenths
        Q = T * 0.1
        tol = 2 * n * n * 2.0 ** -53 * np.abs(Q).sum()  # both sums: n^2 additions of values below sum |Q|
        for r in (h.solve(Q, form=form, tie_rule="qb_f1"), _sharded(h, Q, form, 2), _sharded(h, Q, form, 3)):
            x = X[r["best_X_int"]]
            assert int(x @ T @ x) == lowest
            assert abs(r["best_E"] - 0.1 * lowest) <= tol
