"""The dense route's few-pairs solver at the orders where its quotients' and its bisection's
static and dynamic shared memory pass 48 KB together (n = 1,777 and 3,049) and where the dynamic
part alone does (2,049 and 3,073), and at the largest order it takes, where a thread of the
back-transform holds 32 entries.  What a kernel may ask for is kept by the process, so the
orders run in ascending order in a process of their own: no larger one has gone before.

The matrix is diag(w) between two reflectors, so its eigenvalues are known to the rounding of
three rank-one updates.  Tolerance: ten times n eps |A|, for that and the backward error of
reduction, back-transform and quotients together."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def _check(n, k):
    import numpy as np
    import scipy.sparse as sp
    from conftest import import_package
    s = import_package().speigs
    lib = s.load()
    rng = np.random.default_rng(n)
    w = np.concatenate([0.1 + 0.2 * np.arange(k), 3.0 + rng.random(n - k)])
    A = np.diag(w)
    for _ in range(2):
        v = rng.standard_normal(n)
        v /= np.linalg.norm(v)
        Av = A @ v
        A -= 2.0 * np.outer(v, Av) + 2.0 * np.outer(Av, v) - 4.0 * (v @ Av) * np.outer(v, v)
    A = 0.5 * (A + A.T)
    rc, lam, V, _, info = s.speigs(sp.csc_matrix(A), k, s.SM,
                                   s.default_opts(lib, dense_max=4096, detect=0), lib=lib)
    assert rc == 0, s.last_error(lib)
    assert info["path"] == s.PATH_DENSE and info["nconv"] == k
    bound = 10 * n * np.finfo(float).eps
    assert np.abs(np.sort(lam) - w[:k]).max() <= bound * w.max()
    assert np.linalg.norm(A @ V - V * lam, axis=0).max() <= bound * w.max()
    assert np.abs(V.T @ V - np.eye(k)).max() <= bound


@pytest.mark.parametrize("orders", ["1776,1777,2048,2049", "3048,3049,3072,3073,4096"])
def test_orders_around_the_limits(orders):
    out = subprocess.run([sys.executable, os.path.abspath(__file__), orders],
                         cwd=os.path.dirname(os.path.abspath(__file__)),
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stdout + out.stderr


if __name__ == "__main__":
    for order in sys.argv[1].split(","):
        _check(int(order), 5)
        print("n =", order, "ok", flush=True)
