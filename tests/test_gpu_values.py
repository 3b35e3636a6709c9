"""speigs_plan_set_values through its device map and through the host rebuild: the products,
||A||_1 and a solve after it are those of a plan made from the new values, to the bit, for
every storage the plan accepts."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _matrix(n, rng):
    A = sp.random(n, n, density=min(1.0, 6.0 / n), random_state=np.random.RandomState(rng.integers(1 << 30)))
    A = A + A.T
    return (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 1.0)).tocsc()


def _store(A, how, rng):
    """(n, Ap, Ai, Ax) of A: full or upper, columns sorted or shuffled."""
    M = (sp.triu(A) if how.startswith("upper") else A).tocsc()
    M.sort_indices()
    Ap, Ai, Ax = M.indptr.astype(np.int64), M.indices.astype(np.int64), M.data.copy()
    if how.endswith("shuffled"):
        for c in range(M.shape[0]):
            o = rng.permutation(Ap[c + 1] - Ap[c]) + Ap[c]
            Ai[Ap[c]:Ap[c + 1]], Ax[Ap[c]:Ap[c + 1]] = Ai[o].copy(), Ax[o].copy()
    return M.shape[0], Ap, Ai, Ax


@pytest.mark.parametrize("how", ("full", "upper", "upper shuffled"))
@pytest.mark.parametrize("n", (1, 2, 129, 3000))
def test_new_values_match_a_new_plan(pkg, lib, how, n):
    torch = pytest.importorskip("torch")
    s = pkg.speigs
    rng = np.random.default_rng(n)
    A = _matrix(n, rng)
    args = _store(A, how, rng)
    old = s.Plan(args, s.LM, s.default_opts(lib, check_sym=0), lib=lib)
    x = torch.from_numpy(rng.standard_normal(n)).cuda()
    for step in range(3):
        # new symmetric values on the same pattern, one of them not finite the last time
        f = rng.random(n) + 0.5
        col = np.repeat(np.arange(n), np.diff(args[1]))
        Ax = args[3] * f[args[2]] * f[col]
        if step == 2:
            Ax[(args[2] == n - 1) & (col == n - 1)] = np.nan
        assert old.set_values(Ax) == 0
        new = s.Plan((*args[:3], Ax), s.LM, s.default_opts(lib, check_sym=0), lib=lib)
        y0, y1 = torch.zeros_like(x), torch.ones_like(x)
        torch.cuda.synchronize()
        assert old.apply_device(x.data_ptr(), y0.data_ptr()) == 0
        assert new.apply_device(x.data_ptr(), y1.data_ptr()) == 0
        assert np.array_equal(y0.cpu().numpy(), y1.cpu().numpy(), equal_nan=True)
        if step < 2:
            out = torch.zeros(2 * n + 2, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            infos = [p.solve_device(1, out.data_ptr(), None, None)[1] for p in (old, new)]
            assert infos[0]["anorm"] == infos[1]["anorm"] and infos[0]["nops"] == infos[1]["nops"]
        new.close()
    old.close()
