"""A kernel launch that the runtime refuses becomes an error of the call.

* On the host: the launch wrapper against a stand-in for the runtime's launch call.
* On the GPU: a basis of 12,449 columns, whose Gram-Schmidt coefficients are one column too
  many for a block's shared memory.  The call ends there with SPEIGS_ERR_INTERNAL; it runs in a
  process of its own, under a time limit, and the next call in that process is unharmed."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_wrapper_keeps_the_first_refusal(tmp_path):
    from conftest import PKG_DIR
    exe = tmp_path / "launch_check"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread",
                           "-I", os.path.join(PKG_DIR, "csrc"), "-I/usr/local/cuda/include",
                           os.path.join(HERE, "host", "launch_check.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr


@pytest.mark.gpu
def test_refused_launch_is_an_error():
    out = subprocess.run([sys.executable, os.path.abspath(__file__)], cwd=HERE,
                         capture_output=True, text=True, timeout=240)
    assert out.returncode == 0, out.stdout + out.stderr


def _refused_launch():
    import numpy as np
    import scipy.sparse as sp
    from conftest import import_package
    s = import_package().speigs
    lib = s.load()
    n = 12500
    d, e = np.random.default_rng(1).uniform(1.0, 2.0, n), np.full(n - 1, 1e-3)
    A = sp.diags([e, d, e], [-1, 0, 1]).tocsc()
    rc, *_ = s.speigs(A, 1, s.LM, s.default_opts(lib, ncv=n, maxit=1, detect=0), lib=lib)
    assert rc == s.ERR_INTERNAL and "invalid" in s.last_error(lib), (rc, s.last_error(lib))
    rc, lam, *_ = s.speigs(A, 1, s.LM, s.default_opts(lib, tol=1e-8, detect=0), lib=lib)
    assert rc == 0 and abs(lam[0] - d.max()) < 2e-3


if __name__ == "__main__":
    _refused_launch()
