"""The dense route's few-pairs solver at the orders where its storage changes (one cluster of 8
or 16 blocks, the matrix in shared or in global memory) and on spectra that test the selection
and the clusters: definite, indefinite, repeated and zero eigenvalues, rank one, tiny and huge
scales; against numpy's dense eigensolver."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _matrix(kind, n, rng):
    if kind == "spd":
        B = rng.standard_normal((n, n))
        return B @ B.T / n + np.diag(rng.random(n))
    if kind == "indefinite":
        B = rng.standard_normal((n, n))
        return B + B.T
    if kind == "complete":                       # n - 1 equal eigenvalues and a zero
        return n * np.eye(n) - np.ones((n, n))
    if kind == "rank1":
        v = rng.standard_normal(n)
        return np.outer(v, v)
    if kind == "path":                           # tridiagonal already
        return np.diag(np.full(n, 2.0)) - np.diag(np.ones(n - 1), 1) - np.diag(np.ones(n - 1), -1)
    if kind == "signed":                         # +a and -a pairs
        B = rng.standard_normal((n // 2, n // 2)) + 0.1
        A = np.zeros((n, n))
        A[:n // 2, n // 2:2 * (n // 2)] = B
        return A + A.T
    if kind == "grid":
        m = round(n ** (1 / 3))
        L = _matrix("path", m, rng)
        I = np.eye(m)
        return np.kron(np.kron(L, I), I) + np.kron(np.kron(I, L), I) + np.kron(np.kron(I, I), L)
    raise ValueError(kind)


CASES = ([("spd", n, 6) for n in (23, 24, 25, 65, 128, 210, 256, 257, 463, 468, 640, 660, 800)]
         + [("indefinite", n, 5) for n in (24, 129, 300, 470, 655)]
         + [("complete", 60, 9), ("complete", 300, 12), ("rank1", 100, 4), ("path", 500, 10),
            ("signed", 120, 8), ("signed", 301, 7), ("grid", 216, 20), ("grid", 512, 30),
            ("spd", 100, 64), ("spd", 70, 65), ("spd", 90, 90), ("indefinite", 40, 30)])


@pytest.mark.parametrize("which", ("sm", "lm"))
@pytest.mark.parametrize("case", CASES, ids=str)
def test_pairs_match_numpy(pkg, lib, case, which):
    kind, n, k = case
    s = pkg.speigs
    A = _matrix(kind, n, np.random.default_rng(n + k))
    n = A.shape[0]
    A = 0.5 * (A + A.T)
    rc, lam, V, res, info = s.speigs(sp.csc_matrix(A), k, s.SM if which == "sm" else s.LM,
                                     s.default_opts(lib, dense_max=1000, detect=1), lib=lib)
    assert rc == 0, s.last_error(lib)
    assert info["path"] == s.PATH_DENSE and info["nconv"] == k and info["flag"] == 0
    w = np.linalg.eigvalsh(A)
    want = w[np.argsort(np.abs(w), kind="stable")]
    want = want[:k] if which == "sm" else want[::-1][:k]
    an = np.linalg.norm(A, 2)
    # backward error of the reduction and of numpy's: a small multiple of n eps ||A||; where
    # magnitudes tie to rounding either sign may come first
    tol = 8 * n * np.finfo(float).eps * an
    assert np.max(np.abs(np.abs(lam) - np.abs(want))) <= tol
    assert np.max(np.min(np.abs(lam[:, None] - w[None, :]), axis=1)) <= tol
    assert np.all(np.diff(np.abs(lam)) >= 0) if which == "sm" else np.all(np.diff(np.abs(lam)) <= 0)
    assert np.max(np.linalg.norm(A @ V - V * lam, axis=0)) <= 4 * tol
    assert np.max(np.abs(V.T @ V - np.eye(k))) <= 1e-9
    assert (res == 0).all()


@pytest.mark.parametrize("scale", (1e-120, 1e-90, 1e90, 1e120))
def test_scales(pkg, lib, scale):
    s = pkg.speigs
    A = _matrix("spd", 90, np.random.default_rng(1))
    A = 0.5 * (A + A.T)
    rc, lam, V, _, _ = s.speigs(sp.csc_matrix(A * scale), 4, s.SM, s.default_opts(lib), lib=lib)
    assert rc == 0
    w = np.linalg.eigvalsh(A)[:4]
    assert np.max(np.abs(lam / scale - w)) <= 8 * 90 * np.finfo(float).eps * np.linalg.norm(A, 2)
