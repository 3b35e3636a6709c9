"""Gram-Schmidt passes, Ritz vectors and residuals over every split of rows and
columns: one block, several blocks with a ragged last one, segments that are
split among column groups, more than eight and more than 64 columns, odd row
counts, more vectors than one chunk.  Checked through the largest eigenpairs of
a sparse matrix with a known spectrum: a diagonal with separated top values,
plus a weak chain (norm below 2e-3), against NumPy's dense solver where n is small.

Tolerances: the basis is orthogonalised twice, so that its columns are
orthonormal to a few times the sum of m rounding errors: 1e-12 over all sizes
here; the solver stops at a residual of 1e-10 |A| (its tolerance), checked at
twice that."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,ncv", [
    (40, 3, 12), (513, 1, 3), (1025, 9, 24), (4096, 17, 70), (40001, 5, 20), (151553, 11, 33),
    (700001, 2, 9),
])
def test_lanczos_basis(pkg, lib, n, k, ncv):
    s = pkg.speigs
    rng = np.random.default_rng(n)
    d = rng.uniform(0.0, 1.0, n)
    top = rng.choice(n, k, replace=False)
    d[top] = 2.0 + np.arange(k)[::-1] * 0.5
    e = np.full(n - 1, 1e-3)
    A = sp.diags([e, d, e], [-1, 0, 1]).tocsc()
    A.sort_indices()
    csc = (n, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data.copy())
    rc, lam, V, _, _ = s.speigs(csc, k, s.LM, s.default_opts(lib, tol=1e-10, ncv=ncv), lib=lib)
    assert rc == 0
    lam, V = np.asarray(lam), np.asarray(V)
    V = V if V.shape[0] == n else V.T
    anorm = float(abs(A).sum(axis=0).max())
    assert np.abs(V.T @ V - np.eye(k)).max() <= 1e-12
    assert np.linalg.norm(A @ V - V * lam, axis=0).max() <= 2e-10 * anorm
    assert np.abs(np.sort(lam) - np.sort(d[top])).max() <= 2e-3
