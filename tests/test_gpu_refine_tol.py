"""speigs_ext_opts.refine_tol in a plan's applications, before any solve: the refinement stops at
the caller's backward error, ||r|| <= refine_tol (||A||_1 ||y|| + ||b||), one column or several.

With 1 the first solve is accepted: its error is that of a factor stored in FP32, 6e-8 a rounding,
and stays above 1e-12 however the roundings cancel.  With 1e-15 the error is at most that (NumPy's
own residual adds 1e-16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr", (1, 8))
@pytest.mark.parametrize("tol,lo,hi", ((1.0, 1e-12, 1.0), (1e-9, 0.0, 1e-9), (1e-15, 0.0, 1.1e-15)))
def test_applications_stop_at_the_callers_target(pkg, lib, tol, lo, hi, nr):
    torch = pytest.importorskip("torch")
    s = pkg.speigs
    A = pkg.workloads.varcoef3d(20, seed=5)
    n = A.shape[0]
    plan = s.Plan(A, s.SM, s.default_opts(lib), lib=lib,
                  ext=s.ext_opts(lib, precision=s.MIXED, refine_tol=tol))
    b = torch.from_numpy(np.random.default_rng(nr).standard_normal((nr, n))).cuda()
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    assert plan.factor() == (0, 0.0)
    rc = (plan.apply_device(b.data_ptr(), x.data_ptr()) if nr == 1 else
          plan.apply_block_device(b.data_ptr(), n, x.data_ptr(), n, nr))
    assert rc == 0, s.last_error(lib)
    B, X = b.cpu().numpy().T, x.cpu().numpy().T
    err = np.linalg.norm(B - A @ X, axis=0) / (abs(A).sum(axis=0).max() * np.linalg.norm(X, axis=0) +
                                               np.linalg.norm(B, axis=0))
    assert lo <= err.max() <= hi, err
    plan.close()
