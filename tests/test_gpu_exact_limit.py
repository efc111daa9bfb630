"""The exact form refuses a whole problem of 49 variables (2^33 records) as out of memory."""
import numpy as np
import pytest

import qubo_b200  # noqa: F401
from qubo_b200 import _lib

pytestmark = pytest.mark.gpu


def test_whole_problem_too_large_for_the_exact_form(cuda_ok):
    h = _lib.handle(0)
    with pytest.raises(_lib.QbError, match="device memory allocation failed"):
        h.solve(np.eye(49), form="exact")
    Q = np.diag(np.arange(-5, 15))
    assert h.solve(Q, form="exact")["best_E_int"] == -15  # the handle goes on working
