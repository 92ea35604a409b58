"""Rows of P that end within a round of 128 entries of 2^31, the largest number of entries that is accepted: the
relabelling and the attractive pass, launched alone on arrays of 2^31 entries whose tail alone is filled.

Relabelling: exact. Attraction: FP64 restatement; each lane sums at most two entries a row in FP32 and the warp's sum has
five levels, each term's factors and products are within 6 units of 2^-24: 2^-20 of the sum of magnitudes.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fastembedr_gb300 import _lib, build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ENTRIES, TAIL = 1 << 31, 1024
LAST = ENTRIES - 1  # the largest bound of a row


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    _lib.require_gpu()
    out = str(tmp_path_factory.mktemp("edges") / "kernel_edges.so")
    subprocess.run([build.nvcc(), "-std=c++17", *build.ARCH, "-O3", "-lineinfo", "-shared", "-Xcompiler", "-fPIC",
                    os.path.join(HERE, "kernel_edges.cu"), build.LIB, "-o", out], check=True)
    return C.CDLL(out)


def _rows(bounds):
    return np.array([[LAST - a, LAST - b] for a, b in bounds], np.int32)


# a whole round and part of one, a row within one round, rows beside each other on both sides of a multiple of 4
BOUNDS = [(500, 301), (301, 129), (129, 128), (128, 4), (4, 3), (3, 0), (600, 500), (601, 600)]


def test_relabel(lib):
    rows = _rows(BOUNDS)
    n = len(rows)
    rng = np.random.default_rng(1)
    delta = rng.permutation(n).astype(np.int32)
    col = rng.integers(0, n, TAIL).astype(np.int32)
    want = col.copy()
    for a, b in rows - (ENTRIES - TAIL):
        want[a:b] = delta[want[a:b]]
    assert lib.edge_relabel(rows.ctypes.data_as(C.c_void_p), n, col.ctypes.data_as(C.c_void_p), C.c_longlong(TAIL),
                            delta.ctypes.data_as(C.c_void_p)) == 0
    np.testing.assert_array_equal(col, want)


def test_attractive(lib):
    rows = _rows(BOUNDS)
    n = len(rows)
    rng = np.random.default_rng(2)
    col = rng.integers(0, n, TAIL).astype(np.int32)
    val = rng.uniform(0.0, 1.0, TAIL).astype(np.float32)
    y = rng.normal(size=(n, 2)).astype(np.float32)
    got = np.zeros((n, 2), np.float32)
    assert lib.edge_attractive(rows.ctypes.data_as(C.c_void_p), n, col.ctypes.data_as(C.c_void_p),
                               val.ctypes.data_as(C.c_void_p), C.c_longlong(TAIL), y.ctypes.data_as(C.c_void_p),
                               got.ctypes.data_as(C.c_void_p)) == 0
    y64 = y.astype(np.float64)
    for i, (a, b) in enumerate(rows - (ENTRIES - TAIL)):
        d = y64[i] - y64[col[a:b]]
        t = (val[a:b] / (1 + (d * d).sum(1)))[:, None] * d
        assert (np.abs(got[i] - t.sum(0)) <= 2.0 ** -20 * np.abs(t).sum(0)).all()
