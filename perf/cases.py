"""The solver's work, as its users have it done, for timing and comparison.

Every case goes through the package's public entry points: speigs() on host arrays,
a resident Plan (solves, operator applications, refactorizations), speigs_batched() and
the warm-start network.  The operators are those of the repository's benchmark: finite-volume
diffusion on a box grid with log-normal conductivity (a smooth random field, or independent
cells) and random geometric graphs, all drawn from the seed alone.

Eigenvectors are defined up to their sign; run() fixes it (a positive product with a fixed
vector), so that two correct solvers return the same vectors.  Residual norms and operator
counts are diagnostics of the rounding and are not returned.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sparse-eigs-mex_b200")


def package():
    """The package, imported by path: its folder's name is no Python identifier."""
    if "speigs_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "speigs_b200", os.path.join(PKG, "__init__.py"), submodule_search_locations=[PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["speigs_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["speigs_b200"]


# ------------------------------------------------------------------ cases --
def box(name, kind, dims, field="grf", **more):
    c = {"name": name, "kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "field": field}
    c.update(more)
    return c


def listed():
    return [
        # a small matrix given to the drop-in call once: at most 800 unknowns go to the
        # dense route (the default dense_max); latency
        box("dropin_dense_210", "dropin", (5, 6, 7), k=6, which="sm"),
        # the smallest benchmark operator (20^3) through the drop-in call: ordering, analysis,
        # factor, Lanczos and copies, host arrays to host arrays
        box("dropin_sm_20", "dropin", (20, 20, 20), k=6, which="sm"),
        # a family of operators on one pattern: the matrix and its analysis stay on the GPU,
        # each pass factors and iterates to the k smallest (the benchmark's 46^3)
        box("solve_sm_46_k6", "solve", (46, 46, 46), k=6, which="sm", block=-1, ncv=0),
        # the largest benchmark operator (64^3, independent cells, k = 20)
        box("solve_sm_64_k20", "solve", (64, 64, 64), field="iid", k=20, which="sm", block=-1,
            ncv=0),
        # the benchmark's metric operator (48^3, k = 16) by the block method as it is tuned there
        box("solve_block_48_k16", "solve", (48, 48, 48), k=16, which="sm", block=8, ncv=96),
        # largest eigenvalues: Lanczos on the matrix itself, a million unknowns, no factor
        box("solve_lm_100_k6", "solve", (100, 100, 100), field="iid", k=6, which="lm", block=-1,
            ncv=0),
        # the factored operator as a preconditioner or a propagator: 24 right-hand sides at once
        box("apply24_48", "apply", (48, 48, 48), nr=24, mixed=False),
        # a time step with new coefficients on an odd grid: new values, factor, one solve
        box("refactor_apply1_35", "refactor", (33, 35, 37), nr=1, mixed=False),
        # the same with the FP32 factor and FP64 refinement, 8 right-hand sides
        box("refactor_mixed_apply8_48", "refactor", (48, 48, 48), nr=8, mixed=True),
        # many graphs in one call, k smallest of every connected component
        {"name": "batched_rgg_32", "kind": "batched", "graphs": 32, "nmin": 50, "nmax": 2500,
         "k": 4},
        # the warm-start network's proposal for one operator of the benchmark's size
        box("mpnn_forward_48", "mpnn_forward", (48, 48, 48), nout=24, layers=4),
        # one training step of it: forward, loss, backward (the gradients are read back)
        box("mpnn_train_32", "mpnn_train", (32, 32, 32), nout=24, layers=4, k=16),
    ]


def draw(rng):
    def edges(lo, hi):
        """Three grid sizes with lo <= their geometric mean <= hi, each its own."""
        m = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        a, b = math.exp(rng.uniform(-0.2, 0.2)), math.exp(rng.uniform(-0.2, 0.2))
        return [max(2, round(v)) for v in (m * a, m * b, m / (a * b))]

    def on(kind, dims, **more):
        c = box("", kind, dims, **more)
        del c["name"]
        return c

    kind = rng.choice(["dense", "dropin", "solve", "solve", "block", "lm", "apply", "refactor",
                       "refactor", "batched", "mpnn_forward", "mpnn_train"])
    field = rng.choice(["grf", "iid"])
    if kind == "dense":
        return on("dropin", edges(3.2, 8.8), field=field, k=rng.randint(1, 12), which="sm")
    if kind == "dropin":
        return on("dropin", edges(11, 36), field=field, k=rng.randint(1, 12),
                  which=rng.choice(["sm", "sm", "lm"]) if field == "iid" else "sm")
    if kind == "solve":
        return on("solve", edges(14, 56), field=field, k=rng.randint(1, 20), which="sm",
                  block=-1, ncv=0)
    if kind == "block":
        b = rng.choice([4, 8, 16])
        return on("solve", edges(18, 52), field=field, k=rng.randint(4, 20), which="sm", block=b,
                  ncv=rng.choice([96, 128]))
    if kind == "lm":
        return on("solve", edges(20, 96), field="iid", k=rng.randint(1, 8), which="lm", block=-1,
                  ncv=0)
    if kind == "apply":
        return on("apply", edges(12, 58), field=field, nr=rng.randint(1, 32),
                  mixed=rng.random() < 0.3)
    if kind == "refactor":
        return on("refactor", edges(12, 58), field=field, nr=rng.randint(1, 16),
                  mixed=rng.random() < 0.3)
    if kind == "batched":
        hi = int(math.exp(rng.uniform(math.log(400), math.log(2500))))
        return {"kind": "batched", "graphs": rng.randint(4, 40), "nmin": 50, "nmax": hi,
                "k": rng.randint(1, 6)}
    return on(kind, edges(10, 48 if kind == "mpnn_forward" else 34), nout=rng.choice([16, 24, 32]),
              layers=rng.randint(2, 5), **({"k": rng.randint(4, 16)} if kind == "mpnn_train" else {}))


# ----------------------------------------------------------------- inputs --
def conductivity(case, seed):
    """Cell conductivities exp(g) [z, y, x] on the GPU: g a smooth Gaussian field of unit
    variance and correlation length a tenth of the box (grf), or independent cells (iid)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["field"] == "iid":
        return torch.randn(nz, ny, nx, generator=g, dtype=torch.float64, device="cuda").exp()
    noise = torch.randn(2 * nz, 2 * ny, 2 * nx, generator=g, dtype=torch.float64, device="cuda")
    h = 1.0 / max(nx, ny, nz)
    kz, ky, kx = (2 * math.pi * torch.fft.fftfreq(2 * m, d=h, device="cuda", dtype=torch.float64)
                  for m in (nz, ny, nx))
    k2 = kz[:, None, None] ** 2 + ky[None, :, None] ** 2 + kx[None, None, :] ** 2
    f = torch.fft.ifftn(torch.fft.fftn(noise) * torch.exp(-0.25 * 0.01 * k2)).real
    f = f[:nz, :ny, :nx]
    return ((f - f.mean()) / f.std()).exp()


def faces(kap):
    """Per cell the transmissibilities to its 6 neighbours (-z, -y, -x, +x, +y, +z; 0 where the
    cell has none there) and the diagonal, Dirichlet boundary faces included."""
    T = torch.zeros(6, *kap.shape, dtype=torch.float64, device=kap.device)
    diag = torch.zeros_like(kap)
    for ax in range(3):
        m = kap.shape[ax]
        a, b = kap.narrow(ax, 0, m - 1), kap.narrow(ax, 1, m - 1)
        t = 2 * a * b / (a + b)
        T[ax].narrow(ax, 1, m - 1).copy_(t)
        T[5 - ax].narrow(ax, 0, m - 1).copy_(t)
        for at in (0, m - 1):
            diag.select(ax, at).add_(2 * kap.select(ax, at))
    return T, diag + T.sum(0)


def fv_csc(kap):
    """The finite-volume operator (n, Ap, Ai, Ax): CSC, both triangles, sorted rows, host."""
    T, diag = faces(kap)
    nz, ny, nx = kap.shape
    n = kap.numel()
    off = torch.tensor([-nx * ny, -nx, -1, 0, 1, nx, nx * ny], device=kap.device)
    full = torch.cat([-T[:3].reshape(3, n), diag.reshape(1, n), -T[3:].reshape(3, n)]).t()
    rows = torch.arange(n, device=kap.device)[:, None] + off
    there = full != 0
    Ap = torch.zeros(n + 1, dtype=torch.int64, device=kap.device)
    Ap[1:] = there.sum(1).cumsum(0)
    return n, Ap.cpu().numpy(), rows[there].cpu().numpy(), full[there].cpu().numpy()


def graphs_csc(case, seed):
    """Block-diagonal Laplacians (+ 1e-3 I) of random geometric graphs with about 8 neighbours a
    node: CSC, both triangles, sorted rows, host.  The graphs are the case's, the edge weights
    the seed's."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    at = torch.Generator(device="cuda").manual_seed(case["graphs"] * 10007 + case["nmax"])
    sizes = np.random.default_rng(case["graphs"] * 10007 + case["nmax"]).integers(
        case["nmin"], case["nmax"] + 1, size=case["graphs"])
    R, C, W, base = [], [], [], 0
    for m in (int(v) for v in sizes):
        p = torch.rand(m, 3, generator=at, dtype=torch.float64, device="cuda")
        u = torch.rand(m, generator=g, dtype=torch.float64, device="cuda")
        near = torch.cdist(p, p) < 1.12 * (24.0 / (4.0 * math.pi * m)) ** (1.0 / 3.0)
        near.fill_diagonal_(True)
        r, c = near.nonzero(as_tuple=True)
        w = -(0.5 + 0.5 * (u[r] + u[c]))
        w[r == c] = 0.0
        d = torch.zeros(m, dtype=torch.float64, device="cuda").index_add_(0, r, -w)
        w[r == c] = d + 1e-3
        R.append(r + base)
        C.append(c + base)
        W.append(w)
        base += m
    R, C, W = torch.cat(R), torch.cat(C), torch.cat(W)
    Ap = torch.zeros(base + 1, dtype=torch.int64, device="cuda")
    Ap[1:] = torch.bincount(R, minlength=base).cumsum(0)     # symmetric: row r is column r
    return base, Ap.cpu().numpy(), C.cpu().numpy(), W.cpu().numpy()


def network_inputs(case, seed):
    """Graph (CSR of the normalised adjacency), node features, targets and parameters."""
    kap = conductivity(case, seed)
    T, _ = faces(kap)
    nz, ny, nx = kap.shape
    n = kap.numel()
    s = T.sum(0).reshape(n)
    T = T.reshape(6, n).t()
    off = torch.tensor([-nx * ny, -nx, -1, 1, nx, nx * ny], device="cuda")
    cols = torch.arange(n, device="cuda")[:, None] + off
    there = T != 0
    w = (T / torch.sqrt(s[:, None] * s[cols.clamp(0, n - 1)]))[there].float()
    rp = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    rp[1:] = there.sum(1).cumsum(0).int()
    z, y, x = (torch.arange(1, m + 1, device="cuda", dtype=torch.float64) * math.pi / (m + 1)
               for m in (nz, ny, nx))
    lg = kap.log().reshape(n)
    X = [(lg - lg.mean()) / lg.std()]
    for a, b, c in ((1, 1, 1), (1, 1, 2), (1, 2, 1), (2, 1, 1), (1, 2, 2), (2, 1, 2), (2, 2, 1)):
        v = (torch.sin(a * z)[:, None, None] * torch.sin(b * y)[:, None]
             * torch.sin(c * x)).reshape(n)
        X.append(v / v.norm() * math.sqrt(n))
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    U = None
    if "k" in case:
        U = torch.linalg.qr(torch.randn(n, case["k"], generator=g, dtype=torch.float64,
                                        device="cuda"))[0].float().contiguous()
    par = []
    for o, i in shapes(case):
        par.append(torch.randn(o * i, generator=g, dtype=torch.float64, device="cuda")
                   / math.sqrt(i))
        par.append(0.1 * torch.randn(o, generator=g, dtype=torch.float64, device="cuda"))
    return {"n": n, "rp": rp, "ci": cols[there].int(), "w": w,
            "X": torch.stack(X, 1).float().contiguous(), "U": U,
            "params": torch.cat(par).float().cpu().numpy()}


def shapes(case):
    return [(64, 8)] + [(64, 128)] * case["layers"] + [(case["nout"], 64)]


def rhs(n, nr, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 2)
    return torch.randn(nr, n, generator=g, dtype=torch.float64, device="cuda")


def probe(n):
    """The fixed vector whose product with an eigenvector is made positive."""
    return np.random.default_rng(1).standard_normal(n)


# ------------------------------------------------------- the measured pass --
def prepare(case, seed):
    pkg = package()
    s = pkg.speigs
    lib = s.load()
    kind = case["kind"]
    st = {"case": case, "s": s, "lib": lib}
    if kind == "batched":
        st["A"] = graphs_csc(case, seed)
        st["opts"] = s.default_opts(lib, tol=1e-10)
        st["comp"] = s.components(st["A"], lib)[1]
        st["probe"] = probe(st["A"][0])
        return st
    if kind.startswith("mpnn"):
        st.update(network_inputs(case, seed))
        st["net"] = pkg.learned.WarmStartNet(nout=case["nout"], layers=case["layers"], lib=lib)
        st["net"].set_params(st["params"])
        st["Y"] = torch.empty(st["n"], case["nout"], dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return st
    st["A"] = A = fv_csc(conductivity(case, seed))
    n = A[0]
    if kind == "dropin":
        st["which"] = s.SM if case["which"] == "sm" else s.LM
        st["opts"] = s.default_opts(lib, tol=1e-10)
        st["probe"] = probe(n)
        return st
    if kind == "solve":
        st["plan"] = s.Plan(A, s.SM if case["which"] == "sm" else s.LM,
                            s.default_opts(lib, tol=1e-10, ncv=case["ncv"]), lib=lib,
                            ext=s.ext_opts(lib, block=case["block"]))
        st["lam"] = torch.zeros(case["k"], dtype=torch.float64, device="cuda")
        st["V"] = torch.zeros(case["k"], n, dtype=torch.float64, device="cuda")
        st["probe"] = torch.from_numpy(probe(n)).cuda()
        torch.cuda.synchronize()
        return st
    st["plan"] = s.Plan(A, s.SM, s.default_opts(lib), lib=lib,
                        ext=s.ext_opts(lib, precision=s.MIXED if case["mixed"] else s.FP64))
    st["B"] = rhs(n, case["nr"], seed)
    st["Y"] = torch.zeros_like(st["B"])
    torch.cuda.synchronize()
    if kind == "apply" and st["plan"].factor()[0] != 0:
        raise RuntimeError("factor: " + s.last_error(lib))
    return st


def checked(st, rc):
    if rc != 0:
        raise RuntimeError("%s (%s)" % (st["s"].errmsg(rc, st["lib"]), st["s"].last_error(st["lib"])))


def run(st):
    case, s = st["case"], st["s"]
    kind = case["kind"]
    if kind == "dropin":
        rc, lam, V, _, _ = s.speigs(st["A"], case["k"], st["which"], st["opts"], lib=st["lib"])
        checked(st, rc)
        V *= np.sign(st["probe"] @ V)
        return {"lam": lam, "V": V}
    if kind == "batched":
        rc, lam, V, _, _, _ = s.speigs_batched(st["A"], case["k"], s.SM, st["opts"],
                                               comp=st["comp"], vectors=True, lib=st["lib"])
        checked(st, rc)
        for t in range(case["k"]):
            sign = np.sign(np.bincount(st["comp"], weights=V[:, t] * st["probe"]))
            V[:, t] *= sign[st["comp"]]
        return {"lam": lam, "V": V}
    if kind == "solve":
        rc, _ = st["plan"].solve_device(case["k"], st["lam"].data_ptr(), st["V"].data_ptr(), None)
        checked(st, rc)
        return {"lam": st["lam"], "V": st["V"] * torch.sign(st["V"] @ st["probe"])[:, None]}
    if kind in ("apply", "refactor"):
        p, B, Y, n = st["plan"], st["B"], st["Y"], st["A"][0]
        if kind == "refactor":
            checked(st, p.set_values(st["A"][3]))
            checked(st, p.factor()[0])
        if case["nr"] == 1:
            checked(st, p.apply_device(B.data_ptr(), Y.data_ptr()))
        else:
            checked(st, p.apply_block_device(B.data_ptr(), n, Y.data_ptr(), n, case["nr"]))
        return Y
    net, ptr = st["net"], [st[k].data_ptr() for k in ("rp", "ci", "w", "X")]
    if kind == "mpnn_forward":
        checked(st, net.forward_device(st["n"], *ptr, st["Y"].data_ptr(), 0))
        return st["Y"]
    loss = net.train_step_device(st["n"], *ptr, st["U"].data_ptr(), case["k"], 0.0, 0)
    return {"loss": loss, "grads": net.grads()}


# ------------------------------------------------------------------- work --
def work(case):
    """Inputs read once and outputs written once; the operations are those of a dense eigensolver
    with k vectors, of a nested-dissection factor of a 3-D grid (about 2.6 n^2) and of products
    with it (about 5 n^(4/3) entries), of the network's layers, and of one operator application
    per wanted pair."""
    kind = case["kind"]
    if kind == "batched":
        m = [0.5 * (case["nmin"] + case["nmax"])] * case["graphs"]
        n = sum(m)
        return {"bytes": n * (9 * 16 + 8 + 8 * case["k"]), "flops": sum(2.6 * v ** 2 for v in m)}
    n = case["nx"] * case["ny"] * case["nz"]
    matrix, entries = n * (7 * 16 + 8), 5 * n ** (4 / 3)
    if kind.startswith("mpnn"):
        par = sum(o * i for o, i in shapes(case))
        steps = 3 if kind == "mpnn_train" else 1
        return {"bytes": n * (4 + 6 * 8 + 4 * 8 + 4 * case.get("k", case["nout"])) + 4 * par,
                "flops": steps * n * (2 * par + 2 * 6 * 64 * case["layers"])}
    if kind in ("dropin", "solve"):
        k = case["k"]
        out = 8 * n * k
        if case["which"] == "lm":
            return {"bytes": matrix + out, "flops": 14 * n * k}
        if kind == "dropin" and n <= 800:
            return {"bytes": matrix + out, "flops": 4 / 3 * n ** 3 + 2 * n * n * k}
        return {"bytes": matrix + out, "flops": 2.6 * n * n + 4 * entries * k}
    size = 4 if case["mixed"] else 8
    solve = 4 * entries * case["nr"]
    if kind == "apply":
        return {"bytes": size * entries + 16 * n * case["nr"], "flops": solve}
    return {"bytes": matrix + 16 * n * case["nr"], "flops": 2.6 * n * n + solve}


# ------------------------------------------------------------------ exact --
def sparse(A):
    """The symmetric CSC (n, Ap, Ai, Ax) as a sparse CSR tensor on the GPU."""
    n, Ap, Ai, Ax = A
    return torch.sparse_csr_tensor(torch.from_numpy(Ap).cuda(), torch.from_numpy(Ai).cuda(),
                                   torch.from_numpy(Ax).cuda(), size=(n, n), dtype=torch.float64)


def cg(M, d, B, tol=1e-15):
    """M X = B for the columns of B: conjugate gradients scaled by the diagonal d, restarted from
    the true residual."""
    X = torch.zeros_like(B)
    ref = B.norm(dim=0)
    for _ in range(4):
        R = B - M @ X
        Z = R / d
        P = Z.clone()
        rz = (R * Z).sum(0)
        for it in range(3000):
            Q = M @ P
            a = rz / (P * Q).sum(0).clamp_min(1e-300)
            X += a * P
            R -= a * Q
            Z = R / d
            new = (R * Z).sum(0)
            P = Z + (new / rz.clamp_min(1e-300)) * P
            rz = new
            if it % 25 == 24 and bool((R.norm(dim=0) <= tol * ref).all()):
                break
    return X


def smallest(A, k):
    """The k smallest eigenpairs of a large SPD matrix: block inverse iteration in a growing
    subspace, every solve by conjugate gradients."""
    M = sparse(A)
    n = A[0]
    d = torch.zeros(n, dtype=torch.float64, device="cuda")
    col = np.repeat(np.arange(n), np.diff(A[1]))
    at = np.nonzero(A[2] == col)[0]
    d = torch.from_numpy(A[3][at]).cuda()[:, None]
    g = torch.Generator(device="cuda").manual_seed(3)
    p = k + 8
    W = torch.randn(n, p, generator=g, dtype=torch.float64, device="cuda")
    Q = torch.linalg.qr(W)[0]
    for _ in range(2):
        basis, W = [Q], Q
        for _ in range(5):
            W = cg(M, d, W, 1e-13)
            for _ in range(2):
                for q in basis:
                    W = W - q @ (q.t() @ W)
            W = torch.linalg.qr(W)[0]
            basis.append(W)
        V = torch.cat(basis, 1)
        V = torch.linalg.qr(V)[0]
        w, S = torch.linalg.eigh(V.t() @ (M @ V))
        Q = torch.linalg.qr(V @ S[:, :p])[0]
    V = V @ S[:, :k]
    return w[:k], V / V.norm(dim=0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batched":
        return exact_batched(case, seed)
    if kind.startswith("mpnn"):
        return exact_network(case, seed)
    n = case["nx"] * case["ny"] * case["nz"]
    A = fv_csc(conductivity(case, seed))
    if kind in ("apply", "refactor"):
        col = np.repeat(np.arange(n), np.diff(A[1]))
        d = torch.from_numpy(A[3][A[2] == col]).cuda()[:, None]
        return cg(sparse(A), d, rhs(n, case["nr"], seed).t().contiguous()).t().contiguous()
    if case["which"] == "lm" or n > 70000:
        return None
    k = case["k"]
    if n <= 4000:
        w, V = torch.linalg.eigh(sparse(A).to_dense())
        w, V = w[:k], V[:, :k]
    else:
        w, V = smallest(A, k)
    V = V * torch.sign(torch.from_numpy(probe(n)).cuda() @ V)
    return {"lam": w, "V": V} if kind == "dropin" else {"lam": w, "V": V.t().contiguous()}


def exact_batched(case, seed):
    n, Ap, Ai, Ax = graphs_csc(case, seed)
    k = case["k"]
    lab = np.arange(n)
    col = np.repeat(np.arange(n), np.diff(Ap))
    while True:                                  # the smallest node of each component
        new = lab.copy()
        np.minimum.at(new, col, lab[Ai])
        new = new[new]
        if np.array_equal(new, lab):
            break
        lab = new
    first = np.unique(lab)                       # components in order of first appearance
    comp = np.searchsorted(first, lab)
    order = np.argsort(comp, kind="stable")
    ends = np.cumsum(np.bincount(comp))
    lam, V = np.zeros((len(first), k)), np.zeros((n, k))
    where = np.empty(n, dtype=np.int64)
    prob = probe(n)
    for c, end in enumerate(ends):
        nodes = order[end - np.sum(comp == c):end]
        where[nodes] = np.arange(len(nodes))
        at = np.concatenate([np.arange(Ap[j], Ap[j + 1]) for j in nodes])
        D = torch.zeros(len(nodes), len(nodes), dtype=torch.float64)
        D[where[Ai[at]], where[col[at]]] = torch.from_numpy(Ax[at])
        w, S = torch.linalg.eigh(D.cuda() if len(nodes) > 64 else D)
        m = min(k, len(nodes))
        S = S[:, :m].cpu().numpy()
        lam[c, :m] = w[:m].cpu().numpy()
        V[nodes, :m] = S * np.sign(prob[nodes] @ S)
    return {"lam": lam, "V": V}


def exact_network(case, seed):
    """The network in 64 bits from its 32-bit parameters and inputs."""
    z = network_inputs(case, seed)
    n = z["n"]
    A = torch.sparse_csr_tensor(z["rp"].long(), z["ci"].long(), z["w"].double(), size=(n, n))
    par = torch.from_numpy(z["params"]).double().cuda()
    lay, at = [], 0
    for o, i in shapes(case):
        lay.append((par[at:at + o * i].reshape(o, i), par[at + o * i:at + o * i + o]))
        at += o * i + o
    hs, xs = [torch.tanh(z["X"].double() @ lay[0][0].t() + lay[0][1])], [z["X"].double()]
    for W, b in lay[1:-1]:
        xs.append(torch.cat([hs[-1], A @ hs[-1]], 1))
        hs.append(torch.tanh(xs[-1] @ W.t() + b))
    Y = hs[-1] @ lay[-1][0].t() + lay[-1][1]
    if kind_forward(case):
        return Y
    k, P = case["k"], case["nout"]
    U = z["U"].double()
    G = Y.t() @ Y
    G = G + 1e-8 * torch.trace(G) / P * torch.eye(P, dtype=torch.float64, device="cuda")
    B = Y.t() @ U
    C = torch.linalg.solve(G, B)
    loss = 1.0 - torch.trace(B.t() @ C) / k
    dY = -(2.0 / k) * (U - Y @ C) @ C.t()
    grads = [torch.cat([(dY.t() @ hs[-1]).reshape(-1), dY.sum(0)])]
    dh = dY @ lay[-1][0]
    for l in range(len(lay) - 2, -1, -1):
        dz = dh * (1.0 - hs[l] ** 2)
        grads.append(torch.cat([(dz.t() @ xs[l]).reshape(-1), dz.sum(0)]))
        if l:
            dx = dz @ lay[l][0]
            dh = dx[:, :64] + A @ dx[:, 64:]     # the adjacency is symmetric
    return {"loss": float(loss), "grads": torch.cat(grads[::-1])}


def kind_forward(case):
    return case["kind"] == "mpnn_forward"
