"""The tile solves at the sizes where their tiles can go wrong: fronts around the strip
width (128 columns, one right-hand side; 64 in a block) and the strip height (512 rows; 256 in
a block), every padded width of the block form, leading dimensions above n, and repeated
solves of alternating widths (the values that pass between tasks exist in two copies).  The
right-hand sides and results against the matrix itself, in FP64."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _dense(n, rng):
    B = rng.standard_normal((n, n))
    return sp.csc_matrix(B @ B.T + n * np.eye(n))


def _tree(blocks, sep, rng):
    """`blocks` paths of 40 nodes, each tied to a dense separator of `sep` nodes."""
    n = 40 * blocks + sep
    rows, cols = [], []
    for q in range(blocks):
        for a in range(39):
            rows.append(40 * q + a)
            cols.append(40 * q + a + 1)
        for t in rng.choice(sep, size=min(sep, 9), replace=False):
            rows.append(40 * q + int(rng.integers(40)))
            cols.append(40 * blocks + int(t))
    S = sp.coo_matrix((-rng.random(len(rows)) - 0.1, (rows, cols)), shape=(n, n)).tocsr()
    D = sp.lil_matrix((n, n))
    D[40 * blocks:, 40 * blocks:] = -rng.random((sep, sep))
    S = S + D.tocsr()
    A = S + S.T
    A.setdiag(0)
    return (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 0.2)).tocsc()


MATS = ([("dense", n) for n in (1, 15, 16, 17, 64, 65, 128, 129, 257, 512, 513, 1030)]
        + [("tree", 30, 20), ("tree", 60, 130), ("tree", 20, 300)])


@pytest.mark.parametrize("case", MATS, ids=str)
@pytest.mark.parametrize("mixed", (False, True))
def test_solves_match_the_matrix(pkg, lib, case, mixed):
    torch = pytest.importorskip("torch")
    s = pkg.speigs
    rng = np.random.default_rng(sum(case[1:]))
    A = {"dense": _dense, "tree": _tree}[case[0]](*case[1:], rng)
    A.sort_indices()
    n = A.shape[0]
    p = s.Plan(A, s.SM, s.default_opts(lib), lib=lib,
               ext=s.ext_opts(lib, precision=s.MIXED if mixed else s.FP64))
    assert p.factor()[0] == 0
    an = abs(A).sum(axis=0).max()
    # an n-column Cholesky solve has a normwise backward error of a small multiple of n eps;
    # the mixed form refines to 1e-14 over the whole block
    bound = 4 * n * np.finfo(float).eps + 1e-14
    ld = n + 3
    seen = {}
    for nr in (1, 8, 13, 24, 8, 32, 1, 2, 24, 8):
        B = np.random.default_rng(nr).standard_normal((nr, ld))
        tb = torch.from_numpy(B).cuda()
        ty = torch.full_like(tb, 7.0)
        torch.cuda.synchronize()
        if nr == 1:
            assert p.apply_device(tb.data_ptr(), ty.data_ptr()) == 0
        else:
            assert p.apply_block_device(tb.data_ptr(), ld, ty.data_ptr(), ld, nr) == 0
        Y = ty.cpu().numpy()
        assert (Y[:, n:] == 7.0).all()
        Y = Y[:, :n]
        R = np.linalg.norm((A @ Y.T).T - B[:, :n])
        assert R <= bound * np.sqrt(nr) * (an * np.linalg.norm(Y) + np.linalg.norm(B[:, :n])), nr
        if nr in seen:
            assert np.array_equal(seen[nr], Y), f"width {nr}: two solves differ"
        seen[nr] = Y
    p.close()


def test_infinite_and_nan_right_hand_sides_pass_through(pkg, lib):
    """A value that is not finite reaches the results; no task waits for it."""
    torch = pytest.importorskip("torch")
    s = pkg.speigs
    A = pkg.workloads.lap3d(9)
    n = A.shape[0]
    p = s.Plan(A, s.SM, s.default_opts(lib), lib=lib)
    assert p.factor()[0] == 0
    rng = np.random.default_rng(0)
    for bad in (np.nan, np.inf, np.uint64(0x7ffcb200b200b200).view(np.float64)):
        b = rng.standard_normal((8, n))
        b[3, 100] = bad
        tb, ty = torch.from_numpy(b).cuda(), torch.zeros(8, n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert p.apply_block_device(tb.data_ptr(), n, ty.data_ptr(), n, 8) == 0
        Y = ty.cpu().numpy()
        assert not np.isfinite(Y[3]).any() and np.isfinite(np.delete(Y, 3, axis=0)).all()
        assert p.apply_device(tb[3].data_ptr(), ty.data_ptr()) == 0
        assert not np.isfinite(ty.cpu().numpy()[0]).any()
    p.close()
