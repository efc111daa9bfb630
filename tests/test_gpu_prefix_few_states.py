"""Per-prefix minima of prefixes with few states: warps over several prefixes (B < 5), one (5), parts
of one (6, 7), the first size of the other kernel (8), and problems of fewer states than a warp has
lanes, against all energies in FP64 on the host, integer Q bit-exact."""
import numpy as np
import pytest

import oracle
import qubo_b200  # noqa: F401
from qubo_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,B", [(1, 0), (1, 1), (3, 0), (3, 2), (4, 4), (5, 5), (7, 7), (7, 6), (9, 0), (12, 3), (14, 4),
                                 (14, 5), (15, 6), (16, 7), (16, 8), (18, 1)])
@pytest.mark.parametrize("dtype", [np.int64, np.float32])
def test_prefix_minima_of_few_states(cuda_ok, n, B, dtype):
    rng = np.random.default_rng(64 * n + B)
    Q = (rng.integers(-9, 10, (n, n)) if dtype == np.int64 else rng.standard_normal((n, n))).astype(dtype)
    got = _lib.handle(0).prefix_minima(Q, prefix_bits=n - B)
    want = oracle.prefix_minima_numpy(Q, n - B)
    if dtype == np.int64:
        assert np.array_equal(got, want)
    else:  # both sums have at most n^2 additions of values below sum |Q|
        assert np.abs(got - want).max() <= 2 * n * n * 2.0 ** -53 * np.abs(Q.astype(np.float64)).sum()
