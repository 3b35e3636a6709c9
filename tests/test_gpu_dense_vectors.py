"""The few-pairs solver's back-transform (a block of 128 threads a column, with 2, 8 or 32 entries a
thread up to n = 256, 1,024 and above), its bisection (512 points a round) and its quotients (256
rows at a time, four threads a row) at the orders where a warp, an entry or a chunk of rows or
columns begins.

Tolerances: backward error n eps |A| for the reduction and the back-transform together, with a
factor of ten; the quotients are in twice the precision, so an eigenvalue is off by the square
of its vector's error over the gap: 1e-13 |A| covers it."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [25, 31, 32, 33, 63, 97, 255, 256, 257, 288, 289, 511, 512, 513])
def test_vectors_and_quotients(pkg, lib, n):
    s = pkg.speigs
    rng = np.random.default_rng(n)
    k = 5
    Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    w = np.concatenate([0.1 + 0.2 * np.arange(k), 3.0 + rng.random(n - k)])
    A = (Q * w) @ Q.T
    A = 0.5 * (A + A.T)
    rc, lam, V, _, info = s.speigs(sp.csc_matrix(A), k, s.SM,
                                   s.default_opts(lib, dense_max=1000, detect=1), lib=lib)
    assert rc == 0 and info["path"] == s.PATH_DENSE
    lam, V = np.asarray(lam), np.asarray(V)
    norm = np.abs(w).max()
    exact = np.linalg.eigvalsh(A)[:k]
    assert np.abs(np.sort(lam) - exact).max() <= 1e-13 * norm
    bound = 10 * n * np.finfo(float).eps
    assert np.abs(V.T @ V - np.eye(k)).max() <= bound
    assert np.linalg.norm(A @ V - V * lam, axis=0).max() <= bound * norm
