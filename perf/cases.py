"""Performance cases of the two-site DMRG path.

Each case is one call (or one whole run) that a user of the framework makes: the
effective-Hamiltonian apply, a Lanczos solve, environment updates in both directions,
the two-site splits, the adjoint gradient, and a whole two-site DMRG run, in the plain
FP64 form (the default of every entry point) and in the mixed TF32x3 form.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges,
``prepare(case, seed)`` the inputs on the GPU, ``run(state)`` one pass through the public
entry points, ``work(case)`` the bytes and operations that a pass cannot do without and
``exact(case, seed)`` what ``run`` returns in 64 bits from plain torch.

Inputs are those of a DMRG sweep: environments are contracted from random isometries
(canonical site tensors) and a Hamiltonian MPO, two-site wavefunctions carry decaying
Schmidt weights on their bonds or, for a local solve, lie near its solution.  They come from the seed and plain torch alone.
"""
import ctypes as C
import math

import numpy as np
import torch

import chemtensor_mojo_gb300 as ct
from chemtensor_mojo_gb300.autograd import energy_and_gradient

# MPO bond dimension and physical dimension of the model Hamiltonians
MODELS = {"ising": (3, 2), "xxz": (5, 2), "bose": (4, 4), "hubbard": (6, 4)}
FLOP_CAP = {"fp64": 6.0e9, "tf32x3": 2.2e12}   # of one drawn pass, by precision form


def listed():
    return [
        # the smallest call: one apply on a short chain, where launches and latency count
        dict(name="heff_fp64_16", kind="heff", prec="fp64", model="xxz", Dl=16, Dr=16),
        # the default form at an ordinary bond dimension
        dict(name="heff_fp64_256", kind="heff", prec="fp64", model="xxz", Dl=256, Dr=256),
        # odd bond dimensions, d = 4 (the Fermi-Hubbard chain's MPO), mixed form
        dict(name="heff_mixed_hubbard_odd", kind="heff", prec="tf32x3", model="hubbard", Dl=211, Dr=163),
        # the benchmark chain's centre bond, one apply (a caller with its own eigensolver)
        dict(name="heff_mixed_1024", kind="heff", prec="tf32x3", model="xxz", Dl=1024, Dr=1024),
        # local solve of the L=12 Ising run: 20 steps of the reference's plain Lanczos
        dict(name="lanczos_fp64_32", kind="lanczos", prec="fp64", model="ising", Dl=32, Dr=32, iters=20),
        # local solve of the benchmark chain's centre bond: 24 reorthogonalised steps
        dict(name="lanczos_mixed_1024", kind="lanczos", prec="tf32x3", model="xxz", Dl=1024, Dr=1024, iters=24),
        # environment updates of both half-sweeps: the centre of the benchmark chain ...
        dict(name="env_left_mixed_1024", kind="env", prec="tf32x3", model="xxz", left=True, Dl=1024, Dr=1024),
        # ... and ragged bonds in the default form
        dict(name="env_right_fp64_ragged", kind="env", prec="fp64", model="bose", left=False, Dl=117, Dr=150),
        # exact split with truncation and spectrum (default form), 256 x 256
        dict(name="split_fp64_128", kind="split", model="xxz", Dl=128, Dr=128, left=True),
        # warm split of a bond where chi_max binds: every large bond of a mixed sweep
        dict(name="split_warm_512", kind="warm", model="xxz", Dl=512, Dr=512, left=True),
        # adjoint gradient of every site tensor: the Bose-Hubbard chain, checkpoints every 6 sites
        dict(name="grad_fp64_bose", kind="grad", prec="fp64", model="bose", L=32, chi=128, every=6),
        # a whole mixed-form run: Heisenberg chain in a site-dependent field, two sweeps
        dict(name="dmrg_mixed_heis16", kind="dmrg", prec="tf32x3", L=16, chi=64, sweeps=2, iters=24),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    for _ in range(1000):
        c = _draw(rng)
        if work(c)["flops"] <= FLOP_CAP[c.get("prec", "tf32x3")]:
            return c
    raise RuntimeError("no case drawn")


def _draw(rng):
    kind = rng.choice(["heff", "heff", "lanczos", "lanczos", "env", "env", "split", "warm", "grad", "dmrg"])
    prec = rng.choice(["fp64", "tf32x3"])
    model = rng.choice(sorted(MODELS))
    fp64 = prec == "fp64"
    if kind in ("heff", "env"):
        lo, hi = (8, 256) if fp64 else (48, 1024)
        D = _log_int(rng, lo, hi)
        c = dict(kind=kind, prec=prec, model=model, Dl=D, Dr=min(hi, max(lo, int(D * rng.uniform(0.6, 1.6)))))
        if kind == "env":
            c["left"] = rng.random() < 0.5
        return c
    if kind == "lanczos":
        lo, hi = (8, 64) if fp64 else (64, 1024)
        D = _log_int(rng, lo, hi)
        return dict(kind=kind, prec=prec, model=model, Dl=D, Dr=min(hi, max(lo, int(D * rng.uniform(0.6, 1.6)))),
                    iters=rng.randint(12, 24))
    if kind == "split":
        D = _log_int(rng, 12, 128)
        return dict(kind=kind, model="xxz", Dl=D, Dr=min(128, int(D * rng.uniform(0.8, 1.25))),
                    left=rng.random() < 0.5)
    if kind == "warm":
        D = _log_int(rng, 96, 512)
        return dict(kind=kind, model=rng.choice(["xxz", "hubbard"]) if D <= 256 else "xxz", Dl=D,
                    Dr=min(512, int(D * rng.uniform(0.8, 1.25))), left=rng.random() < 0.5)
    if kind == "grad":
        return dict(kind=kind, prec=prec, model=model, L=rng.randint(6, 32), chi=_log_int(rng, 8, 128),
                    every=rng.choice([0, 4, 6]))
    return dict(kind="dmrg", prec=prec, L=rng.randint(8, 14), chi=rng.randint(16, 64), sweeps=2,
                iters=rng.randint(16, 24))


# ---- Hamiltonian MPOs (W[wl, in, out, wr]) ------------------------------------------------
def _bulk(model):
    """-> (bulk tensor, channel that starts a term, channel that has finished one)."""
    D, d = MODELS[model]
    if model in ("ising", "xxz"):
        X, Z = np.array([[0.0, 1.0], [1.0, 0.0]]), np.diag([1.0, -1.0])
        P, M = np.array([[0.0, 1.0], [0.0, 0.0]]), np.array([[0.0, 0.0], [1.0, 0.0]])
        I = np.eye(2)
        if model == "ising":
            e = {(0, 0): I, (1, 0): -Z, (2, 0): -X, (2, 1): Z, (2, 2): I}
        else:
            e = {(0, 0): I, (1, 0): 0.5 * M, (2, 0): 0.5 * P, (3, 0): 0.25 * Z, (4, 1): P, (4, 2): M, (4, 3): Z,
                 (4, 4): I}
    elif model == "bose":
        b = np.diag(np.sqrt(np.arange(1.0, d)), 1)
        n = np.diag(np.arange(float(d)))
        e = {(0, 0): np.eye(d), (1, 0): -b, (2, 0): -b.T, (3, 0): 2.0 * n @ (n - np.eye(d)), (3, 1): b.T, (3, 2): b,
             (3, 3): np.eye(d)}
    else:
        cu, cd = np.zeros((4, 4)), np.zeros((4, 4))
        cu[1, 0] = cu[3, 2] = cd[2, 0] = 1.0
        cd[3, 1] = -1.0
        p = np.diag([1.0, -1.0, -1.0, 1.0])
        e = {(0, 0): np.eye(4), (5, 0): 8.0 * np.diag([0.0, 0.0, 0.0, 1.0]), (5, 5): np.eye(4)}
        for k, (lo, ro) in enumerate([(cu @ p, cu.T), (cd @ p, cd.T), (p @ cu.T, cu), (p @ cd.T, cd)]):
            e[(5, k + 1)] = lo
            e[(k + 1, 0)] = -ro
    W = np.zeros((D, d, d, D))
    for (l, r), op in e.items():
        W[l, :, :, r] = op
    return W, D - 1, 0


def _chain(model, L):
    W, s, f = _bulk(model)
    return [W[s:s + 1]] + [W] * (L - 2) + [W[:, :, :, f:f + 1]]


def _heisenberg_in_field(L, seed):
    """Heisenberg chain with a site-dependent field (no degenerate Schmidt values)."""
    rng = np.random.default_rng(seed)
    sites = [W.copy() for W in _chain("xxz", L)]
    for i, W in enumerate(sites):
        h = rng.uniform(-0.5, 0.5) * np.diag([0.5, -0.5])
        W[-1, :, :, 0] -= h
    return sites


# ---- inputs -------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float64, device="cuda")


def _isometry(g, Dl, d, Dr):
    """Left-canonical site [Dl, d, Dr] (Dl d >= Dr): orthonormal columns over (Dl, d)."""
    q, r = torch.linalg.qr(_randn(g, Dl * d, Dr))
    return (q * torch.sign(torch.diagonal(r))).reshape(Dl, d, Dr).contiguous()


def _left_step(L, A, W):
    """[wL, Dl, Dl'] -> [wR, Dr, Dr']."""
    t = torch.einsum("wab,asc->wbsc", L, A)
    t = torch.einsum("wbsc,wstv->vcbt", t, W)
    return torch.einsum("vcbt,btd->vcd", t, A).contiguous()


def _right_step(R, A, W):
    """[wR, Dr, Dr'] -> [wL, Dl, Dl']."""
    t = torch.einsum("vcd,asc->vasd", R, A)
    t = torch.einsum("vasd,wstv->watd", t, W)
    return torch.einsum("watd,btd->wab", t, A).contiguous()


def _solved(g, theta, L, R, W):
    """theta after a few single-precision Lanczos runs, plus a little noise: the wavefunction
    that a sweep brings to a bond it has visited before is close to the solution."""
    Lf, Rf, Wf = L.float(), R.float(), W.float()
    v = theta.float()
    for _ in range(3):
        V = [v.reshape(-1) / v.norm()]
        al, be = [], []
        for j in range(12):
            w = _heff(V[j].reshape(theta.shape), Lf, Rf, Wf).reshape(-1)
            al.append(float(w @ V[j]))
            if j == 11:
                break
            for _ in range(2):
                B = torch.stack(V)
                w = w - B.T @ (B @ w)
            be.append(float(w.norm()))
            if be[-1] < 1e-4 * abs(al[0]):
                be.pop()
                break
            V.append(w / be[-1])
        c = np.linalg.eigh(np.diag(al) + np.diag(be, 1) + np.diag(be, -1))[1][:, 0]
        v = sum(float(ci) * x for ci, x in zip(c, V)).reshape(theta.shape)
    v = v.double() / v.norm()
    return (v + 1e-2 * theta / theta.norm()).contiguous()


def _dims_to(D, d):
    dims = [1]
    while dims[-1] < D:
        dims.append(min(dims[-1] * d, D))
    return dims


def _left_env(g, model, D):
    W, s, _ = _bulk(model)
    W = torch.from_numpy(W).cuda()
    d = W.shape[1]
    L = torch.ones(1, 1, 1, dtype=torch.float64, device="cuda")
    dims = _dims_to(D, d)
    if len(dims) == 1:
        dims = [1, 1]
    for i in range(len(dims) - 1):
        L = _left_step(L, _isometry(g, dims[i], d, dims[i + 1]), W[s:s + 1] if i == 0 else W)
    return L


def _right_env(g, model, D):
    W, _, f = _bulk(model)
    W = torch.from_numpy(W).cuda()
    d = W.shape[1]
    R = torch.ones(1, 1, 1, dtype=torch.float64, device="cuda")
    dims = _dims_to(D, d)
    if len(dims) == 1:
        dims = [1, 1]
    for i in range(len(dims) - 1):
        A = _isometry(g, dims[i], d, dims[i + 1]).permute(2, 1, 0).contiguous()   # right-canonical
        R = _right_step(R, A, W[:, :, :, f:f + 1] if i == 0 else W)
    return R


def _theta(g, Dl, d, Dr):
    """Normalised two-site wavefunction with Schmidt weights decaying along both bonds."""
    wl = torch.exp(-6.0 * torch.arange(Dl, dtype=torch.float64, device="cuda") / Dl)
    wr = torch.exp(-6.0 * torch.arange(Dr, dtype=torch.float64, device="cuda") / Dr)
    t = _randn(g, Dl, d, d, Dr) * wl[:, None, None, None] * wr
    return (t / t.norm()).contiguous()


def _split_inputs(g, Dl, d, Dr):
    """theta = U diag(s) V^T with a decaying spectrum (about 5e-5 of the weight past half the
    states) -> (theta as a matrix, V)."""
    m, n = Dl * d, d * Dr
    k = min(m, n)
    U = torch.linalg.qr(_randn(g, m, k))[0]
    V = torch.linalg.qr(_randn(g, n, k))[0]
    s = torch.exp(-10.0 * torch.arange(k, dtype=torch.float64, device="cuda") / k)
    s = s / s.norm()
    return ((U * s) @ V.T).contiguous(), U, V


def _inputs(case, seed):
    """The case's arrays as plain torch tensors."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "dmrg":
        L, d = case["L"], 2
        W = [torch.from_numpy(np.ascontiguousarray(w)).cuda() for w in _heisenberg_in_field(L, seed)]
        dims = [min(2 ** i, 2 ** (L - i), 16) for i in range(L + 1)]
        A = [_isometry(g, dims[i + 1], d, dims[i]).permute(2, 1, 0).contiguous() for i in range(L)]
        A[0] = A[0] / A[0].norm()
        return dict(W=W, A=A)
    model = case["model"]
    D, d = MODELS[model]
    if kind == "grad":
        L, chi = case["L"], case["chi"]
        dims = [min(d ** min(i, 16), d ** min(L - i, 16), chi) for i in range(L + 1)]
        A = [_randn(g, dims[i], d, dims[i + 1]) / math.sqrt(dims[i] * d) for i in range(L)]
        return dict(W=[torch.from_numpy(np.ascontiguousarray(w)).cuda() for w in _chain(model, L)], A=A)
    Dl, Dr = case["Dl"], case["Dr"]
    if kind == "split":
        return dict(M=_split_inputs(g, Dl, d, Dr)[0])
    if kind == "warm":
        M, U, V = _split_inputs(g, Dl, d, Dr)
        c = min(Dl, Dr)
        B = V if case["left"] else U
        X = torch.linalg.qr(B[:, :c] + 1e-5 * _randn(g, B.shape[0], c))[0]
        X = X * torch.sign((X * B[:, :c]).sum(0))
        return dict(M=M, X=X.T.contiguous(), c=c)
    W = torch.from_numpy(_bulk(model)[0]).cuda()
    if kind == "env":
        if case["left"]:
            return dict(W=W, E=_left_env(g, model, Dl), A=_isometry(g, Dl, d, Dr) if Dl * d >= Dr
                        else _randn(g, Dl, d, Dr) / math.sqrt(Dl * d))
        A = (_isometry(g, Dr, d, Dl).permute(2, 1, 0).contiguous() if Dr * d >= Dl
             else _randn(g, Dl, d, Dr) / math.sqrt(d * Dr))
        return dict(W=W, E=_right_env(g, model, Dr), A=A)
    L, R, theta = _left_env(g, model, Dl), _right_env(g, model, Dr), _theta(g, Dl, d, Dr)
    return dict(W=W, L=L, R=R, theta=_solved(g, theta, L, R, W) if kind == "lanczos" else theta)


def _dt(t):
    return ct.DenseTensor(t.contiguous().reshape(-1), list(t.shape))


def prepare(case, seed):
    x = _inputs(case, seed)
    ctx = ct.get_context()
    st = dict(case=case, ctx=ctx)
    kind = case["kind"]
    if kind in ("heff", "lanczos"):
        st.update(L=_dt(x["L"]), R=_dt(x["R"]), theta=_dt(x["theta"]), W=ct.MPOSite(_dt(x["W"])))
    elif kind == "env":
        st.update(E=_dt(x["E"]), A=ct.MPSSite(_dt(x["A"])), W=ct.MPOSite(_dt(x["W"])))
    elif kind == "split":
        d = MODELS[case["model"]][1]
        st.update(theta=_dt(x["M"].reshape(case["Dl"], d, d, case["Dr"])))
    elif kind == "warm":
        m, n = x["M"].shape
        c = x["c"]
        new = lambda k: torch.empty(k, dtype=torch.float64, device="cuda")
        st.update(M=x["M"], X=x["X"], c=c, basis=new(c * (m if case["left"] else n)), A=new(m * c), B=new(c * n))
    elif kind == "grad":
        st.update(mpo=ct.MatrixProductOperator([ct.MPOSite(_dt(w)) for w in x["W"]]), sites=x["A"])
    else:
        st.update(mpo=ct.MatrixProductOperator([ct.MPOSite(_dt(w)) for w in x["W"]]),
                  mps=ct.MatrixProductState([ct.MPSSite(_dt(a)) for a in x["A"]]))
    return st


def run(st):
    case, ctx = st["case"], st["ctx"]
    kind = case["kind"]
    if kind == "heff":
        return ct.apply_two_site_heff(st["theta"], st["L"], st["R"], st["W"], st["W"], ctx,
                                      prec=case["prec"]).storage
    if kind == "lanczos":
        # converged tridiagonal eigensolve; the mixed form reorthogonalises, as in its sweeps
        E, v = ct.lanczos_two_site_optimize(st["theta"], st["L"], st["R"], st["W"], st["W"], ctx,
                                            max_iter=case["iters"], tol=1e-10, prec=case["prec"], max_rotations=0,
                                            reorth=case["prec"] == "tf32x3")
        return E, v.storage
    if kind == "env":
        f = ct.update_left_environment if case["left"] else ct.update_right_environment
        return f(st["E"], st["A"], st["W"], ctx, prec=case["prec"]).storage
    if kind == "split":
        A, B, disc, S = ct.split_two_site_theta_svd(st["theta"], min(case["Dl"], case["Dr"]), 1e-10, ctx,
                                                    left_to_right=case["left"], return_spectrum=True)
        return A.tensor.storage, B.tensor.storage, disc, S
    if kind == "warm":
        d = MODELS[case["model"]][1]
        ok, disc = C.c_int(), C.c_double()
        p = lambda t: C.c_void_p(t.data_ptr())
        ctx.call("ct_svd_split_warm", p(st["M"]), C.c_int64(case["Dl"]), C.c_int64(d), C.c_int64(case["Dr"]),
                 C.c_int64(st["c"]), int(case["left"]), p(st["X"]), 0, p(st["basis"]), p(st["A"]), p(st["B"]),
                 C.byref(ok), C.byref(disc), None)
        return ok.value, disc.value, st["basis"], st["A"], st["B"]
    if kind == "grad":
        E, grads = energy_and_gradient(st["mpo"], st["sites"], case["every"], ctx, prec=case["prec"])
        return [E] + list(grads)
    p = ct.DMRGParams(num_sweeps=case["sweeps"], chi_max=case["chi"], eps_trunc=0.0, max_krylov_iter=case["iters"],
                      krylov_tol=1e-10, energy_tol=0.0, prec=case["prec"], max_rotations=0, final_rayleigh=True)
    stats = ct.DMRGStats()
    E, mps = ct.dmrg_two_site(ctx, st["mpo"], st["mps"], p, stats)
    return E, stats.energy_rayleigh, stats.sweep_energies, ct.mps_to_statevector(mps, ctx).storage


# ---- the work a pass cannot do without ----------------------------------------------------
def _heff_flops(Dl, d, Dr, w):
    return (2.0 * Dl * w * d * d * Dr * Dl + 4.0 * Dl * d * Dr * w * d * d * w + 2.0 * Dl * d * d * Dr * w * Dr)


def _env_flops(Dl, d, Dr, w):
    return 2.0 * Dl * w * d * Dr * Dl + 2.0 * Dl * Dr * w * d * d * w + 2.0 * w * Dr * Dr * Dl * d


def work(case):
    kind = case["kind"]
    w, d = MODELS[case.get("model", "xxz")]
    if kind in ("heff", "lanczos"):
        Dl, Dr = case["Dl"], case["Dr"]
        n = Dl * d * d * Dr
        it = case.get("iters", 1)
        f = it * _heff_flops(Dl, d, Dr, w)
        if kind == "lanczos":   # alpha, recurrence, norm; the basis twice per step where it is reorthogonalised
            f += it * 10.0 * n + (2.0 * it * it * n if case["prec"] == "tf32x3" else 0.0)
        return dict(bytes=8.0 * (2 * n + w * Dl * Dl + w * Dr * Dr + 2 * w * w * d * d), flops=f)
    if kind == "env":
        Dl, Dr = case["Dl"], case["Dr"]
        f = _env_flops(Dl, d, Dr, w) if case["left"] else _env_flops(Dr, d, Dl, w)
        return dict(bytes=8.0 * (w * Dl * Dl + w * Dr * Dr + Dl * d * Dr + w * w * d * d), flops=f)
    if kind in ("split", "warm"):
        m, n = case["Dl"] * d, case["Dr"] * d
        c = min(case["Dl"], case["Dr"])
        k = min(m, n)
        if kind == "split":
            return dict(bytes=8.0 * (m * n + m * c + c * n + c), flops=4.0 * m * n * k + 8.0 * k ** 3)
        q, o = (m, n) if case["left"] else (n, m)
        return dict(bytes=8.0 * (m * n + m * c + c * n + c * (m + n)),
                    flops=2.0 * c * m * n * 2 + 2.0 * c * c * q + 2.0 * m * n * c + c ** 3)
    if kind == "grad":
        L, chi = case["L"], case["chi"]
        dims = [min(d ** min(i, 16), d ** min(L - i, 16), chi) for i in range(L + 1)]
        f = b = 0.0
        for i in range(L):
            for ww in (w, 1):
                f += _env_flops(dims[i], d, dims[i + 1], ww) * (3 if case["every"] else 2)
                f += 2.0 * dims[i] * ww * d * dims[i + 1] * (dims[i] + dims[i + 1]) + \
                    2.0 * dims[i] * dims[i + 1] * (ww * d) ** 2
            b += 16.0 * dims[i] * d * dims[i + 1]
        return dict(bytes=b, flops=f)
    L, chi = case["L"], case["chi"]
    w, d = MODELS["xxz"]
    dims = [min(2 ** i, 2 ** (L - i), chi) for i in range(L + 1)]
    f = 0.0
    for i in range(L - 1):
        f += 2 * case["sweeps"] * (case["iters"] * _heff_flops(dims[i], d, dims[i + 2], w) +
                                   _env_flops(dims[i], d, dims[i + 1], w))
    return dict(bytes=8.0 * sum(2 * dims[i] * d * dims[i + 1] for i in range(L)) + 8.0 * 2 ** L, flops=f)


# ---- what run() returns, in 64 bits and plain torch -----------------------------------------
def _heff(theta, L, R, W):
    t = torch.einsum("wab,astc->bwstc", L, theta)
    t = torch.einsum("bwstc,wsum->bmutc", t, W)
    t = torch.einsum("bmutc,mtpv->bupvc", t, W)
    return torch.einsum("bupvc,vcd->bupd", t, R).contiguous()


def exact(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "heff":
        return _heff(x["theta"], x["L"], x["R"], x["W"]).reshape(-1)
    if kind == "env":
        return (_left_step if case["left"] else _right_step)(x["E"], x["A"], x["W"]).reshape(-1)
    if kind == "lanczos":
        shape = x["theta"].shape
        V = [x["theta"].reshape(-1) / x["theta"].norm()]
        al, be = [], []
        for j in range(case["iters"]):
            w = _heff(V[j].reshape(shape), x["L"], x["R"], x["W"]).reshape(-1)
            al.append(float(w @ V[j]))
            if j + 1 == case["iters"]:
                break
            for _ in range(2):
                for v in V:
                    w = w - (w @ v) * v
            be.append(float(w.norm()))
            V.append(w / be[-1])
        T = np.diag(al) + np.diag(be, 1) + np.diag(be, -1)
        lam, U = np.linalg.eigh(T)
        c = U[:, 0] if U[:, 0].sum() >= 0 else -U[:, 0]
        y = sum(float(ci) * v for ci, v in zip(c, V))
        return float(lam[0]), y / y.norm()
    if kind == "split":
        s2 = torch.linalg.svdvals(x["M"]) ** 2
        c = min(case["Dl"], case["Dr"])
        tail = (s2.sum() - torch.cumsum(s2, 0)) / s2.sum()
        c = min(c, int((tail > 1e-10).sum()) + 1)
        return None, None, float(s2[c:].sum() / s2.sum()), s2[:c].sqrt()
    if kind == "warm":
        M = x["M"]
        Z = x["X"] @ (M.T if case["left"] else M)
        q, r = torch.linalg.qr(Z.T)
        Q = (q * torch.sign(torch.diagonal(r))).T.contiguous()
        A, B = (Q.T.contiguous(), Q @ M) if case["left"] else (M @ Q.T, Q)
        disc = float(((M - A @ B) ** 2).sum() / (M ** 2).sum())
        return 1, disc, Q.reshape(-1), A.reshape(-1), B.reshape(-1)
    if kind == "grad":
        A = [a.clone().requires_grad_(True) for a in x["A"]]
        one = torch.ones(1, 1, 1, dtype=torch.float64, device="cuda")
        I = torch.eye(MODELS[case["model"]][1], dtype=torch.float64, device="cuda")[None, :, :, None]
        H = N = one
        for a, W in zip(A, x["W"]):
            H, N = _left_step(H, a, W), _left_step(N, a, I)
        E = H.reshape(()) / N.reshape(())
        E.backward()
        return [float(E.detach())] + [a.grad for a in A]
    return None
