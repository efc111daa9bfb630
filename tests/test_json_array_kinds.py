"""Arrays of numpy's subclasses keep their values in the JSON text, bare and inside an object, and
the text is the standard encoder's (CPU)."""
import json

import numpy as np
import pytest

import qubo_b200  # noqa: F401
from qubo_b200 import _json
from qubo_b200.abc import ProblemABC


class Tagged(np.ndarray):
    pass


class Holder(ProblemABC):
    def __init__(self, Q):
        self.Q = Q

    def build_Q_matrix(self, use_gpu=False):
        return np.asarray(self.Q)


def _kind(kind, tmp_path):
    a = np.arange(9, dtype=np.float32).reshape(3, 3)
    if kind == "matrix":
        return np.matrix(a)
    if kind == "memmap":
        m = np.memmap(tmp_path / "q.bin", dtype=a.dtype, mode="w+", shape=a.shape)
        m[:] = a
        return m
    if kind == "masked":
        return np.ma.masked_array(a, mask=a > 7)
    return a.view(Tagged)


@pytest.mark.parametrize("kind", ["matrix", "memmap", "masked", "subclass"])
def test_array_subclasses(kind, tmp_path):
    if _json._jsonpickle is not None:
        pytest.skip("jsonpickle is installed and writes the text")
    Q = _kind(kind, tmp_path)
    plain = np.asarray(Q)
    assert np.array_equal(_json.decode(_json.encode(Q)), plain)
    assert np.array_equal(_json.decode(_json.encode({"q": [Q]}))["q"][0], plain)
    assert np.array_equal(_json.decode(Holder(Q).to_json()).Q, plain)
    for o in (Q, [Q], {"a": {"b": Q}}, Holder(Q)):
        assert _json.encode(o) == json.dumps(_json._enc(o), indent=4)
