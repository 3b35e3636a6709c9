"""Solves with rows that gather the updates of many children: stars and graphs of a few hubs, at
list lengths around the one from which many threads share a list (16), around a warp's and a
block's strides and of thousands, in pivot rows and in rows below them, for every width the
solve kernel has.

Bound: the backward error of the other solve tests, 1e-14 of |A|_1 |x| + |b|.  Solves are the
same to the bit when repeated.  A star's solve may cost ten times a path's of the same order (one
row's list is 20,000 entries long; one after the other they cost a hundred times)."""
import time

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _laplacian(n, i, j, rng):
    W = sp.coo_matrix((rng.random(len(i)) + 0.5, (i, j)), shape=(n, n)).tocsc()
    W = W + W.T
    A = (sp.diags(np.asarray(W.sum(axis=1)).ravel() + 0.01) - W).tocsc()
    A.sort_indices()
    return A


def _graph(kind, rng):
    if kind[0] == "star":
        n = kind[1] + 1
        return _laplacian(n, np.zeros(n - 1, int), np.arange(1, n), rng)
    hubs, leaves = kind[1:]                      # leaf t at hub 0 and, ever more rarely, the next
    I, J = [np.arange(hubs - 1)], [np.arange(1, hubs)]
    for h in range(hubs):
        t = np.arange(0, leaves, 1 << min(h, 12)) + hubs
        I.append(np.full(len(t), h))
        J.append(t)
    return _laplacian(hubs + leaves, np.concatenate(I), np.concatenate(J), rng)


@pytest.mark.parametrize("kind", [("star", 60), ("star", 64), ("star", 65), ("star", 180),
                                  ("star", 6000), ("hubs", 9, 300), ("hubs", 10, 5000),
                                  ("hubs", 70, 3000)], ids=str)
def test_solves(pkg, lib, kind):
    torch = pytest.importorskip("torch")
    s = pkg.speigs
    rng = np.random.default_rng(sum(kind[1:]))
    A = _graph(kind, rng)
    n = A.shape[0]
    anorm = abs(A).sum(axis=0).max()
    plan = s.Plan(A, s.SM, s.default_opts(lib), lib=lib)
    assert plan.factor() == (0, 0.0)
    for nr in (1, 5, 16, 24, 32):
        B = rng.standard_normal((nr, n))
        b = torch.from_numpy(B).cuda()
        got = []
        for _ in range(2):
            x = torch.zeros_like(b)
            torch.cuda.synchronize()
            rc = (plan.apply_device(b.data_ptr(), x.data_ptr()) if nr == 1 else
                  plan.apply_block_device(b.data_ptr(), n, x.data_ptr(), n, nr))
            assert rc == 0, s.last_error(lib)
            got.append(x.cpu().numpy())
        assert np.array_equal(got[0], got[1])
        R = B.T - A @ got[0].T
        assert np.max(np.linalg.norm(R, axis=0) / (anorm * np.linalg.norm(got[0], axis=1) +
                                                   np.linalg.norm(B, axis=1))) <= 1e-14
    plan.close()


def test_a_long_list_costs_little(pkg, lib):
    torch = pytest.importorskip("torch")
    s = pkg.speigs
    rng = np.random.default_rng(0)
    n = 20001
    best = {}
    for kind, i in (("star", np.zeros(n - 1, int)), ("path", np.arange(n - 1))):
        plan = s.Plan(_laplacian(n, i, np.arange(1, n), rng), s.SM, s.default_opts(lib), lib=lib)
        assert plan.factor() == (0, 0.0)
        b = torch.ones(n, dtype=torch.float64, device="cuda")
        x = torch.zeros_like(b)
        torch.cuda.synchronize()
        t = []
        for _ in range(20):
            t0 = time.perf_counter()
            assert plan.apply_device(b.data_ptr(), x.data_ptr()) == 0
            t.append(time.perf_counter() - t0)
        best[kind] = min(t)
        plan.close()
    assert best["star"] <= 10 * best["path"], best
