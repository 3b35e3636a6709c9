"""The supernodes of a clique with a leaf at each of its vertices (host only): a tall front with
many small children.

Bound, from the merging rule.  A leaf's column has 2 entries, so it may be merged at will only
into a front of at most 96 * 2 = 192 rows; the fronts above that, the clique's first D - 192
vertices, may hold 5 % zeros, and what is left fits a triangle of 2 * 192 columns (192 of the
clique and their leaves).  The clique is one supernode but for those."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import PKG_DIR

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def sizes(tmp_path_factory):
    so = tmp_path_factory.mktemp("symbolic") / "probe.so"
    host = os.path.join(PKG_DIR, "csrc", "host")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-pthread", "-shared", "-fPIC", "-I", host,
                           os.path.join(HERE, "host", "symbolic_probe.cpp"),
                           os.path.join(host, "symbolic.cpp"), "-o", str(so)])
    lib = ctypes.CDLL(str(so))

    def run(A):
        A = A.tocsr()
        A.sort_indices()
        rp, ci = A.indptr.astype(np.int64), A.indices.astype(np.int32)
        out = np.zeros(4, np.int64)
        assert lib.symbolic_sizes(A.shape[0], rp.ctypes.data_as(ctypes.c_void_p),
                                  ci.ctypes.data_as(ctypes.c_void_p),
                                  out.ctypes.data_as(ctypes.c_void_p)) == 0
        return dict(zip(("supernodes", "levels", "entries", "exact"), out.tolist()))

    return run


@pytest.mark.parametrize("d", [300, 700, 1500])
def test_leaves_stay_out_of_a_tall_front(sizes, d):
    leaf = sp.identity(d)
    got = sizes(sp.bmat([[np.ones((d, d)), leaf], [leaf, leaf]]))
    assert got["entries"] <= got["exact"] / 0.95 + 384 * 385 // 2, got
    assert got["levels"] <= 2 + 192, got
