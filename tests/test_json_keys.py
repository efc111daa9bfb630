"""Dictionary keys that become the same text are one entry in the JSON, as with the standard
encoder (CPU)."""
import json

import pytest

import qubo_b200  # noqa: F401
from qubo_b200 import _json


@pytest.mark.parametrize("o", [{1: "a", "1": "b"}, {"x": {None: [1], "None": [2]}}, {2.0: 1, "2.0": {}, 3: []}])
def test_keys_of_equal_text(o):
    if _json._jsonpickle is not None:
        pytest.skip("jsonpickle is installed and writes the text")
    assert _json.encode(o) == json.dumps(_json._enc(o), indent=4)
