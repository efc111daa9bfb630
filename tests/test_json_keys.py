"""Dictionary keys that become the same text are one entry in the JSON, as with the standard
encoder, and encoding keeps nothing (CPU)."""
import json

import numpy as np
import pytest

import qubo_b200  # noqa: F401
from qubo_b200 import _json


@pytest.mark.parametrize("o", [{1: "a", "1": "b"}, {"x": {None: [1], "None": [2]}}, {2.0: 1, "2.0": {}, 3: []}])
def test_keys_of_equal_text(o):
    if _json._jsonpickle is not None:
        pytest.skip("jsonpickle is installed and writes the text")
    assert _json.encode(o) == json.dumps(_json._enc(o), indent=4)


def test_nothing_is_kept_per_dtype():
    def kept():
        return sum(len(v) for v in vars(_json).values() if isinstance(v, (dict, list, set)) and v is not vars(_json)["__builtins__"])

    before = kept()
    for w in range(1, 200):
        _json.encode(np.zeros(1, dtype=f"U{w}"))
    assert kept() == before
