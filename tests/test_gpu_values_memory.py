"""New values for a plan when the device has no memory left for the value map: the host rebuilds
the matrix, as it does for columns that are not sorted, and a later call makes the map."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_new_values_without_device_memory(pkg, lib):
    torch = pytest.importorskip("torch")
    import scipy.sparse as sp
    s = pkg.speigs
    n = 1_500_000                                # map 54 MB, values 108 MB
    e = np.ones(n)
    A = sp.diags([e, e, e, e, e, e, e, e, e], range(-4, 5), shape=(n, n), format="csc")
    A.sort_indices()
    args = (n, A.indptr.astype(np.int64), A.indices.astype(np.int64), A.data)
    plan = s.Plan(args, s.LM, s.default_opts(lib, check_sym=0), lib=lib)
    x = torch.ones(n, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    want = np.asarray(abs(A).sum(axis=1)).ravel()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (80 << 20), dtype=torch.uint8, device="cuda")
    for scale in (2.0, 3.0):
        assert plan.set_values(scale * A.data) == 0, s.last_error(lib)
        assert plan.apply_device(x.data_ptr(), y.data_ptr()) == 0
        assert np.array_equal(y.cpu().numpy(), scale * want)
        fill = None                              # there is room for the second call
        torch.cuda.empty_cache()
    plan.close()
