"""The tile factorization at the sizes where its 64 x 64 tiles can go wrong: dense
matrices (one front of n pivots), arrows (few pivots, many rows below them) and banded
matrices around the tile edges, in both storage precisions, against the backward error of
the solution in FP64."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _arrow(head, tail, rng):
    """`tail` dense columns coupled to `head` leaves of 3 nodes each."""
    n = 3 * head + tail
    A = sp.lil_matrix((n, n))
    for q in range(head):
        for a in range(3):
            for b in range(3):
                A[3 * q + a, 3 * q + b] = -0.3
            A[3 * q + a, 3 * head + int(rng.integers(tail))] = -1.0
    A[3 * head:, 3 * head:] = -rng.random((tail, tail))
    A = A.tocsr()
    A = A + A.T
    A.setdiag(0)
    return (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 0.5)).tocsc()


def _dense(n, rng):
    B = rng.standard_normal((n, n))
    return sp.csc_matrix(B @ B.T + n * np.eye(n))


def _band(n, w, rng):
    A = sp.diags([rng.random(n - d) - 1.5 for d in range(1, w + 1)], range(1, w + 1), shape=(n, n))
    A = A + A.T
    return (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 0.1)).tocsc()


CASES = ([("dense", n) for n in (1, 2, 7, 8, 9, 63, 64, 65, 72, 127, 128, 129, 191, 260)]
         + [("arrow", h, t) for h, t in ((30, 5), (40, 64), (40, 65), (200, 130), (10, 193))]
         + [("band", 500, 3), ("band", 700, 64), ("band", 900, 65), ("band", 900, 130)])


@pytest.mark.parametrize("case", CASES, ids=str)
@pytest.mark.parametrize("mixed", (False, True))
def test_factor_backward_error(pkg, lib, case, mixed):
    torch = pytest.importorskip("torch")
    s = pkg.speigs
    rng = np.random.default_rng(sum(case[1:]))
    A = {"dense": _dense, "arrow": _arrow, "band": _band}[case[0]](*case[1:], rng)
    A.sort_indices()
    n = A.shape[0]
    p = s.Plan(A, s.SM, s.default_opts(lib), lib=lib,
               ext=s.ext_opts(lib, precision=s.MIXED if mixed else s.FP64))
    for _ in range(2):                                   # the second reuses the plan's storage
        rc, shift = p.factor()
        assert rc == 0 and shift == 0.0, s.last_error(lib)
    b = rng.standard_normal(n)
    x = torch.from_numpy(b).cuda()
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    assert p.apply_device(x.data_ptr(), y.data_ptr()) == 0
    y = y.cpu().numpy()
    an = abs(A).sum(axis=0).max()
    # an n-column Cholesky solve has a normwise backward error of a small multiple of n eps;
    # the mixed form refines to the same level (its target is 1e-14)
    bound = 4 * n * np.finfo(float).eps + 1e-14
    assert np.linalg.norm(A @ y - b) <= bound * (an * np.linalg.norm(y) + np.linalg.norm(b))
    p.close()


def test_indefinite_tile_is_reported(pkg, lib):
    """A pivot that fails deep inside a front ends the factorization, and the plan goes on to
    the indefinite route with the exact eigenvalues."""
    s = pkg.speigs
    rng = np.random.default_rng(3)
    A = _dense(150, rng).toarray()
    A[100, 100] -= 4 * 150.0 * 2
    rc, lam, _, _, info = s.speigs(sp.csc_matrix(A), 3, s.SM, s.default_opts(lib, dense_max=0, tol=1e-10),
                                   lib=lib)
    assert rc == 0 and info["path"] == s.PATH_LU
    w = np.linalg.eigvalsh(A)
    w = w[np.argsort(abs(w))][:3]
    assert np.allclose(np.sort(lam), np.sort(w), rtol=1e-9)
