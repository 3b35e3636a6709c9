"""The warm-start network's layer kernels (messages gathered into the
tensor-core product, register-tiled backward products) on graphs that are no
grid: nodes without neighbours, degrees around and above the eight edges that
are read at once, node counts around the 64- and 128-node tiles, every
feature and output width that changes a path.  The reference is FP64 with
BF16 rounding where the device rounds (weights, activations, messages).

Tolerances: the two then differ by FP32 sums and by activations that round to
the other BF16 neighbour, 2^-8 of one entry each.  FP32 sums of 128 terms are
off by about 1e-6 of their size, so fewer than one activation in a hundred
flips: below 2^-8 / sqrt(100) = 4e-4 of the output's norm a layer, 2e-3 over
five.  The gradient multiplies that by the square root of the small Gram
system's condition, which orthonormal output weights keep near ten: 2e-2."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _graph(n, seed):
    """Symmetric, irregular: degrees 0 to about 24, unsorted weights of both signs."""
    rng = np.random.default_rng(seed)
    pull = np.where(rng.random(n) < 0.2, 0.0, rng.random(n) ** 3 * 12.0)
    m = int(2.5 * n)
    p = (pull + 1e-9) / (pull + 1e-9).sum()
    i, j = rng.choice(n, m, p=p), rng.choice(n, m, p=p)
    A = sp.coo_matrix((rng.uniform(-0.5, 0.5, m), (i, j)), shape=(n, n))
    A = (A + A.T).tocsr()
    A.sort_indices()
    A.data = A.data.astype(np.float32).astype(np.float64)
    return A


def _reference(torch, params, A, X, dims, U=None):
    F, H, L, P = dims
    rnd = lambda t: t.float().bfloat16().double()
    At = torch.from_numpy(A.toarray())
    p = torch.from_numpy(params.astype(np.float64))
    shapes = [(H, F)] + [(H, 2 * H)] * L + [(P, H)]
    Ws, bs, off = [], [], 0
    for o, i in shapes:
        Ws.append(rnd(p[off:off + o * i].reshape(o, i)))
        bs.append(p[off + o * i:off + o * i + o])
        off += o * i + o
    xs, hs = [torch.from_numpy(X.astype(np.float64))], []
    hs.append(rnd(torch.tanh(xs[0] @ Ws[0].T + bs[0])))
    for l in range(1, L + 1):
        xs.append(torch.cat([hs[-1], rnd(At @ hs[-1])], 1))
        hs.append(rnd(torch.tanh(xs[-1] @ Ws[l].T + bs[l])))
    xs.append(hs[-1])
    Y = hs[-1] @ Ws[-1].T + bs[-1]
    if U is None:
        return Y.numpy()
    Ut = torch.from_numpy(U.astype(np.float64))
    k = U.shape[1]
    G = Y.T @ Y
    G = G + 1e-8 * torch.trace(G) / P * torch.eye(P, dtype=torch.float64)
    B = Y.T @ Ut
    C = torch.linalg.solve(G, B)
    loss = 1.0 - float((B * C).sum()) / k
    dZ = -(2.0 / k) * (Ut - Y @ C) @ C.T
    grads = []
    for l in range(L + 1, -1, -1):
        grads = [(dZ.T @ xs[l]).reshape(-1), dZ.sum(0)] + grads
        if l == 0:
            break
        dx = dZ @ Ws[l]
        dh = dx if l == L + 1 else dx[:, :H] + At.T @ dx[:, H:]
        dZ = dh * (1.0 - hs[l - 1] ** 2)
    return Y.numpy(), loss, torch.cat(grads).numpy()


CASES = [  # n, F, L, P, k
    (1, 1, 1, 4, 0), (127, 64, 0, 12, 4), (128, 9, 1, 64, 0), (129, 9, 2, 7, 5),
    (300, 9, 1, 16, 16), (65, 9, 4, 8, 3), (1000, 9, 3, 24, 12), (257, 5, 0, 6, 2),
]


@pytest.mark.parametrize("n,F,L,P,k", CASES)
def test_layers_match_rounded_reference(pkg, n, F, L, P, k):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(100 + n)
    A = _graph(n, n)
    X = (2.0 * rng.standard_normal((n, F))).astype(np.float32)
    net = pkg.learned.WarmStartNet(nout=P, layers=L, nfeat=F, seed=5)
    params = net.get_params()
    params[-P:] = rng.uniform(-0.1, 0.1, P)
    params[-P - P * 64:-P] = np.linalg.qr(rng.standard_normal((64, P)))[0].T.reshape(-1)
    net.set_params(params)
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
         (A.indptr.astype(np.int32), np.append(A.indices, 0).astype(np.int32),
          np.append(A.data, 0).astype(np.float32), X)]
    ptr = [a.data_ptr() for a in t]
    # straight into the caller's rows, and into rows that are not 16-byte aligned
    out = torch.full((n * P + 9,), 7.0, dtype=torch.float32, device="cuda")
    ref = _reference(torch, params, A, X, (F, 64, L, P))
    for at in (4, 5):
        out.fill_(7.0)
        torch.cuda.synchronize()
        assert net.forward_device(n, *ptr, out.data_ptr() + 4 * at, 0) == 0
        torch.cuda.synchronize()
        got = out.double().cpu().numpy()
        Y = got[at:at + n * P].reshape(n, P)
        assert np.linalg.norm(Y - ref) <= 2e-3 * np.linalg.norm(ref)
        assert (got[:at] == 7.0).all() and (got[at + n * P:] == 7.0).all()
    if k:
        U, _ = np.linalg.qr(rng.standard_normal((n, k)))
        U = U.astype(np.float32)
        tU = torch.from_numpy(U).cuda()
        torch.cuda.synchronize()
        loss = net.train_step_device(n, *ptr, tU.data_ptr(), k, 0.0, 0)
        _, loss_r, grads = _reference(torch, params, A, X, (F, 64, L, P), U)
        assert abs(loss - loss_r) <= 2e-2 * abs(loss_r)
        got = net.grads().astype(np.float64)
        assert np.linalg.norm(got - grads) <= 2e-2 * np.linalg.norm(grads)
