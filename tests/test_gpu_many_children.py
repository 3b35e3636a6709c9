"""Fronts with thousands of small children: the children's update matrices of one to four rows are
loaded 32 at a time.  Stars (one row each), a hub graph's (one to four rows, next to some of up to
ten, which take the general path) and a clique with pendant paths, against SciPy's solver.

Bound: backward error 1e-14 of |A|_1 |x| + |b|, and 1e-13 for the FP32 factor's refined solves.  The
factor of a star of 20,001 vertices may cost thirty times a path's of the same order (one child
after the other it costs seventy times)."""
import time

import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_long_lists import _graph, _laplacian

pytestmark = pytest.mark.gpu


def _clique(m, pendants, rng):
    """A clique of m vertices; pendant t hangs on 1 + t % 4 of them."""
    I, J = np.triu_indices(m, 1)
    I, J = [I], [J]
    for t in range(pendants):
        k = 1 + t % 4
        I.append((np.arange(k) * 7 + t) % m)
        J.append(np.full(k, m + t))
    return _laplacian(m + pendants, np.concatenate(I), np.concatenate(J), rng)


@pytest.mark.parametrize("mixed", (False, True))
@pytest.mark.parametrize("kind", [("star", 3000), ("hubs", 10, 4000), ("clique", 70, 2000),
                                  ("clique", 200, 999)], ids=str)
def test_factor(pkg, lib, kind, mixed):
    torch = pytest.importorskip("torch")
    s = pkg.speigs
    rng = np.random.default_rng(sum(kind[1:]))
    A = _clique(*kind[1:], rng) if kind[0] == "clique" else _graph(kind, rng)
    n = A.shape[0]
    plan = s.Plan(A, s.SM, s.default_opts(lib), lib=lib,
                  ext=s.ext_opts(lib, precision=s.MIXED if mixed else s.FP64))
    B = rng.standard_normal((8, n))
    b = torch.from_numpy(B).cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    assert plan.factor() == (0, 0.0)
    assert plan.apply_block_device(b.data_ptr(), n, x.data_ptr(), n, 8) == 0, s.last_error(lib)
    X = x.cpu().numpy()
    R = B.T - A @ X.T
    assert np.max(np.linalg.norm(R, axis=0) / (abs(A).sum(axis=0).max() * np.linalg.norm(X, axis=1) +
                                               np.linalg.norm(B, axis=1))) <= (1e-13 if mixed else 1e-14)
    plan.close()


def test_many_children_cost_little(pkg, lib):
    s = pkg.speigs
    rng = np.random.default_rng(0)
    n = 20001
    best = {}
    for kind, i in (("star", np.zeros(n - 1, int)), ("path", np.arange(n - 1))):
        plan = s.Plan(_laplacian(n, i, np.arange(1, n), rng), s.SM, s.default_opts(lib), lib=lib)
        t = []
        for _ in range(10):
            t0 = time.perf_counter()
            assert plan.factor() == (0, 0.0)
            t.append(time.perf_counter() - t0)
        best[kind] = min(t)
        plan.close()
    assert best["star"] <= 30 * best["path"], best
