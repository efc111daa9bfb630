"""The one-pass encoder writes the text the standard encoder writes for the same object (CPU), and
the batch descriptors' fast address path falls back for what the buffer protocol refuses."""
import json

import numpy as np
import pytest

import qubo_b200  # noqa: F401
from qubo_b200 import _json, _lib
from qubo_b200.problems import Just_Q, MaxCut, RandomQUBO, ReducedProblem, TSP

OBJECTS = [{}, [], {"a": {}}, {"a": [], "b": [[1, [2.5]]]}, {1: 2, (1, 2): 3}, None, True, 7, "ü\n\"x\"",
           {"device": "cuda", "x": float("inf"), "s": {"q", "p"}, "t": (1, (2,)), "n": np.int16(3)},
           np.zeros((0, 2)), np.array(3.0), np.zeros((2, 2, 2), np.int8), np.zeros(3, dtype=">f4"),
           [{"z": np.eye(2)}], Just_Q(np.eye(3, dtype=np.float32)), RandomQUBO.init_random_instance(1, 5, dtype=np.int16),
           MaxCut.init_random_instance(1, 6), TSP.init_random_instance(1, 3), ReducedProblem(Just_Q(np.eye(4)), [1, 0])]


@pytest.mark.parametrize("k", range(len(OBJECTS)))
@pytest.mark.parametrize("indent", [4, 1, None])
def test_same_text(k, indent):
    if _json._jsonpickle is not None:
        pytest.skip("jsonpickle is installed and writes the text")
    assert _json.encode(OBJECTS[k], indent=indent) == json.dumps(_json._enc(OBJECTS[k]), indent=indent)


def test_batch_descriptors():
    ro = np.eye(4, dtype=np.float32)
    ro.setflags(write=False)
    plain = [np.eye(3, dtype=np.int8), np.eye(1), np.arange(9, dtype=np.int64).reshape(3, 3)]
    odd = [ro, np.asfortranarray(np.arange(9.0).reshape(3, 3)), np.arange(16.0).reshape(4, 4)[::2, ::2], [[1, 2], [3, 4]]]
    for Qs in (plain, odd, plain + odd, []):
        probs, ns, keep = _lib.Handle._batch_problems(Qs)
        assert len(probs) == len(ns) == len(keep) == len(Qs)
        for p, n, k, Q in zip(probs, ns, keep, Qs):
            assert np.array_equal(k, Q) and k.flags.c_contiguous
            assert (p.n, p.ldq, p.q, p.dtype) == (n, n, k.__array_interface__["data"][0], _lib._DTYPES[k.dtype])
    for bad, err in ((np.zeros((2, 3)), ValueError), (np.zeros((2, 2), ">f4"), TypeError), (np.eye(2, dtype=np.uint8), TypeError)):
        with pytest.raises(err):
            _lib.Handle._batch_problems([np.eye(2), bad])
