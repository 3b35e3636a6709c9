"""Ritz vectors and Gram-Schmidt passes at the basis sizes where a kernel's static and dynamic
shared memory pass 48 KB together: Ritz vectors of 120, 184, 248, 376 and 760 columns (wanted
pairs in the residual test, k + 5 in the restart, single vectors and blocks), dot products of
1,023 and 1,024 columns.

The matrix is tridiagonal: a uniformly distributed diagonal and a weak chain, whose largest
values take several restarts; its eigenvalues come from SciPy's tridiagonal solver.  The solver
stops at a residual of 1e-10 |A|, which bounds an eigenvalue's error too; both are checked at
twice that, the orthonormality at 1e-9 (residual over the wanted values' gaps)."""
import numpy as np
import pytest
import scipy.linalg as la
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _matrix(n):
    rng = np.random.default_rng(n)
    d, e = rng.uniform(1.0, 2.0, n), np.full(n - 1, 1e-3)
    A = sp.diags([e, d, e], [-1, 0, 1]).tocsc()
    A.sort_indices()
    return A, la.eigh_tridiagonal(d, e, eigvals_only=True)


def _check(A, lam, V, want):
    anorm = float(abs(A).sum(axis=0).max())
    assert np.abs(np.sort(lam) - np.sort(want)).max() <= 2e-10 * anorm
    assert np.linalg.norm(A @ V - V * lam, axis=0).max() <= 2e-10 * anorm


@pytest.mark.parametrize("ncv,k", [(120, 44), (120, 38), (184, 20), (248, 12), (376, 10), (760, 3)])
def test_ritz_vectors(pkg, lib, ncv, k):
    s = pkg.speigs
    A, w = _matrix(2001)
    rc, lam, V, _, info = s.speigs(A, k, s.LM, s.default_opts(lib, tol=1e-10, ncv=ncv, detect=0),
                                   lib=lib)
    assert rc == 0, s.last_error(lib)
    assert info["nconv"] == k and info["flag"] == 0
    _check(A, lam, V, w[-k:])
    assert np.abs(V.T @ V - np.eye(k)).max() <= 1e-9


@pytest.mark.parametrize("ncv,k", [(120, 38), (120, 44)])
def test_ritz_vectors_of_blocks(pkg, lib, ncv, k):
    s = pkg.speigs
    A, w = _matrix(2001)
    rc, lam, V, _, info, einfo = s.speigs_ex(
        A, k, s.SM, s.default_opts(lib, tol=1e-10, ncv=ncv, detect=0),
        s.ext_opts(lib, block=8), lib=lib)
    assert rc == 0, s.last_error(lib)
    assert einfo["block"] == 8 and info["nconv"] == k and info["flag"] == 0
    _check(A, lam, V, w[:k])


def test_gram_schmidt_of_a_thousand_columns(pkg, lib):
    """Every pair of a matrix of order 1,026 from a basis as large as it: a pass left out at any
    width leaves pairs unconverged."""
    s = pkg.speigs
    n = 1026
    A, w = _matrix(n)
    rc, lam, V, _, info = s.speigs(
        A, n, s.LM, s.default_opts(lib, tol=1e-10, ncv=n, maxit=1, dense_max=0, detect=0), lib=lib)
    assert rc == 0, s.last_error(lib)
    assert info["nconv"] == n and info["flag"] == 0 and info["restarts"] == 0
    _check(A, lam, V, w)
