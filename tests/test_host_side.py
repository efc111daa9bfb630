"""Host side of the library that needs no GPU (csrc/qb_host.cuh), through a g++ harness."""
import ctypes
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "evo-quantum-qubolib_b200", "csrc")
CUDA_INC = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.isdir(CUDA_INC):
        pytest.skip("g++ or the CUDA headers are not available")
    out = str(tmp_path_factory.mktemp("host") / "host_side.so")
    # a load from an address that its type does not allow stops the process
    subprocess.run([gxx, "-std=c++17", "-O1", "-fPIC", "-shared", "-fsanitize=alignment",
                    "-fsanitize-undefined-trap-on-error", "-I", CSRC,
                    "-I", CUDA_INC, os.path.join(HERE, "host_side_harness.cpp"), "-o", out], check=True)
    return ctypes.CDLL(out)


# --- the key under which a captured batch graph is replayed ------------------------------
NAMES = ("problems", "w_doubles", "arena_bytes", "cap", "gtab_items", "units", "selections", "tc_runs", "sm_gtab",
         "sm_gray", "sm_exact", "sm_tc", "any_gray", "tc_pair", "tc_n_max")
FIELDS = len(NAMES) + 9 + 9


def _key(harness, fields):
    f = (ctypes.c_uint64 * FIELDS)(*fields)
    out = (ctypes.c_uint64 * 64)()
    k = harness.h_batch_graph_key(f, FIELDS, out, 64)
    assert 0 < k <= 64
    return list(out[:k])


def test_every_field_is_in_the_key(harness):
    base = list(range(1, FIELDS + 1))
    for i in range(FIELDS):
        other = list(base)
        other[i] += 1000
        assert _key(harness, other) != _key(harness, base)


def _shape(sizes, gl, sms=148):
    """The fields of a batch of integer problems that take the 16-bit pair kernel from 24
    variables and the exact form below 20 (restated from qb_solve_batch's planning)."""
    tc = [n for n in sizes if n >= 24]
    total = sum(1 << (n - 15 - gl.get(n, 5)) for n in tc)
    per = -(-total // min(sms, total))
    items, runs, left = 0, 1, per
    for n in tc:
        groups, g = 1 << (n - 15 - gl.get(n, 5)), 0
        while g < groups:
            take = min(left, groups - g)
            items, g, left = items + 1, g + take, left - take
            if left == 0:
                runs, left = runs + 1, per
    runs += left != per
    pre = sum(1 << (n - min(n, 16)) for n in sizes if n < 20)
    smem = max((n * n + 1 + max(0, f - 13) * 288 + n * (n + 1) // 2) * 8
               for n, f in [(n, gl.get(n, 5) + 12 if n >= 24 else min(n, 16)) for n in sizes])
    return dict(problems=len(sizes), w_doubles=sum(n * n for n in sizes), arena_bytes=items, cap=pre + 4096,
                selections=len(tc), tc_runs=runs, sm_exact=smem, tc_pair=1, tc_n_max=max(tc), sm_tc=121 * 1024)


def test_batches_that_differ_in_the_largest_size_alone(harness):
    """With wider records tuned for 26 variables, these two batches agree in everything but the
    largest n, by which the search kernel lays out its shared memory: a replay of one's graph for
    the other would write W over the barriers behind it."""
    a, b = _shape([26, 32, 9], {26: 8}), _shape([26, 33, 4], {26: 8})
    assert {k for k in a if a[k] != b[k]} == {"tc_n_max"}
    keys = [_key(harness, [s.get(n, 0) for n in NAMES] + [0] * 18) for s in (a, b)]
    assert keys[0] != keys[1]


# --- the exact form's limit ---------------------------------------------------------------
@pytest.mark.parametrize("n", range(20, 63))
def test_exact_form_limit(harness, n):
    """Whole problems beyond the 2^32 records whose results (24 bytes each) a 180 GB GPU can hold
    are refused, as they are when every record's result is kept."""
    harness.h_exact_form_fits.argtypes = [ctypes.c_uint64]
    records = 1 << (n - 16)
    assert harness.h_exact_form_fits(records) == (records * 24 <= 180 << 30)


# --- matrices in host memory ----------------------------------------------------------------
LOAD = """
import ctypes, sys
import numpy as np
L = ctypes.CDLL(sys.argv[1])
L.h_load.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int64, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
n, ld, off, dt = int(sys.argv[2]), int(sys.argv[3]), int(sys.argv[4]), np.dtype(sys.argv[5])
code = 1 + ["f4", "f8", "i1", "i2", "i4", "i8"].index(sys.argv[5])
rng = np.random.default_rng(n)
raw = np.zeros(n * ld * dt.itemsize + 16, np.uint8)
raw = raw[(-raw.ctypes.data) % 8:]  # 8-byte aligned start
Q = raw[off:off + n * ld * dt.itemsize].view(dt).reshape(n, ld)
Q[:] = rng.integers(-50, 50, (n, ld)) if dt.kind == "i" else rng.standard_normal((n, ld))
W, out = np.zeros((n, n)), np.zeros(2)
assert L.h_load(Q.ctypes.data, n, ld, code, W.ctypes.data, out.ctypes.data) == 0
D = Q[:, :n].astype(np.float64)
want = D + D.T
want[np.arange(n), np.arange(n)] = np.diag(D)
assert np.array_equal(W, want) and abs(out[0] - np.abs(D).sum()) <= 1e-12 * out[0] and out[1] == (dt.kind == "i")
"""


# the offset in bytes from an aligned address; a leading dimension of n and beyond
@pytest.mark.parametrize("dt,off", [("f4", 0), ("f4", 2), ("f8", 0), ("f8", 4), ("f8", 1), ("i1", 1), ("i2", 1), ("i4", 3),
                                    ("i8", 4)])
@pytest.mark.parametrize("n,ld", [(1, 1), (7, 9), (62, 62), (62, 65)])
def test_host_matrix_at_any_address(harness, dt, off, n, ld):
    p = subprocess.run([sys.executable, "-c", LOAD, harness._name, str(n), str(ld), str(off), dt], capture_output=True,
                       text=True)
    assert p.returncode == 0, p.stderr


# --- buffers that grow on demand --------------------------------------------------------------
def _grow(harness, room, sizes):
    a, used = (ctypes.c_uint64 * len(sizes))(*sizes), (ctypes.c_uint64 * len(sizes))()
    harness.h_grow(ctypes.c_uint64(room), a, len(sizes), used)
    return list(used)


def test_buffers_grow_by_little(harness):
    big = 150 << 30
    assert _grow(harness, 1 << 40, [1, 4000, 4500, 5000]) == [256, 4500, 4500, 5625]
    assert all(u <= s + (16 << 20) for s, u in zip([1 << 30, big], _grow(harness, 1 << 40, [1 << 30, big])))
    # what fits is not refused for the sake of spare room
    assert _grow(harness, big, [big]) == [big]
    assert _grow(harness, 1000, [1000, 999]) == [1000, 1000]
    assert _grow(harness, 1000, [1001, 900]) == [0, 900]
