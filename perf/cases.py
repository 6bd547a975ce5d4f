"""The work that users of pyinla_gb300 have it do, as cases that can be timed.

Every case goes through a public entry point: the Serinv-named functions
(``pyinla_gb300.algs``), the drop-in solver (``GB300SerinvSolver``), the batch
(``BtaBatch``) and the model classes.  Block matrices are seeded diagonally dominant BTA
matrices; models are SPDE (x) AR(1) fields on regular meshes with Gaussian or count
observations, the sizes those of this repository's benchmark and tests.
"""
import math

import numpy as np
import torch

F64 = torch.float64


# ------------------------------------------------------------------------- the cases
def listed():
    return [
        # one small system factored and solved: the smallest call, launches and host work
        dict(name="tiny_factor_solve", kind="plain", nt=3, b=20, a=2, nrhs=1, selinv=False, host=False),
        # the plain-solve workload: factor, logdet, solve, selected inverse of 2052 rows
        dict(name="plain_nt16_b128", kind="plain", nt=16, b=128, a=4, nrhs=1, selinv=True, host=False),
        # the same calls on NumPy buffers (a program on the host's arrays), ragged tiles
        dict(name="numpy_nt24_b100", kind="plain", nt=24, b=100, a=3, nrhs=1, selinv=True, host=True),
        # block-tridiagonal prior (no arrow): factor, logdet, several right-hand sides, inverse
        dict(name="bt_nt60_b333", kind="bt", nt=60, b=333, a=0, nrhs=3),
        # repeated solves with one factor (samples, predictions): the two sweeps alone
        dict(name="sweeps_nt96_b768", kind="sweeps", nt=96, b=768, a=6, nrhs=1),
        # sparse matrices on the host through the drop-in solver, every call of one evaluation
        dict(name="dropin_24x24_nt48", kind="dropin", side=24, mside=24, nt=48, nb=6, obs=40000),
        # an objective evaluation inside an optimiser's line search (small ragged mesh)
        dict(name="objective_20x17_nt50", kind="objective", side=20, mside=17, nt=50, nb=3, obs=20000, nv=1, grad=False),
        # the benchmark's model: objective and adjoint gradient of one optimiser step
        dict(name="gradient_32x32_nt128", kind="objective", side=32, mside=32, nt=128, nb=6, obs=200000, nv=1, grad=True),
        # trivariate coregional model, the largest blocks: objective and gradient
        dict(name="gradient_coreg3_nt24", kind="objective", side=32, mside=32, nt=24, nb=3, obs=90000, nv=3, grad=True),
        # variances of the latent field and of the linear predictor after a run
        dict(name="marginals_coreg2_nt32", kind="marginals", side=24, mside=16, nt=32, nb=2, obs=20000, nv=2),
        # count data: the inner Newton iteration, one factorization per step
        dict(name="poisson_16x16_nt32", kind="laplace", side=16, mside=16, nt=32, nb=2, obs=8000),
        # the Q(theta) of a small gradient stencil in one captured launch, mixed sizes
        dict(name="batch9_mixed", kind="batch", shapes="256x64x2,256x128x4,512x32x4,512x64x2,768x32x8,256x32x8,512x32x2,768x64x4,300x40x3"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ones' ranges: block edges 20..1100 (3072 for coregional
    models), 3..128 time blocks, arrows of 0..16."""
    kind = rng.choice(["plain", "plain", "bt", "sweeps", "objective", "objective", "objective", "dropin",
                       "marginals", "laplace", "batch"])
    if kind in ("plain", "bt", "sweeps"):
        b = _logint(rng, 20, 1100)
        nt = max(3, min(_logint(rng, 3, 128), int(6.0e8 / b ** 2.4)))
        case = dict(kind=kind, nt=nt, b=b, a=0 if kind == "bt" else rng.randint(1, 16), nrhs=rng.randint(1, 5))
        if kind == "plain":
            case.update(selinv=rng.random() < 0.7, host=b * b * nt < 2e6 and rng.random() < 0.4)
        return case
    if kind == "batch":
        n = rng.randint(3, 12)
        return dict(kind=kind, shapes=",".join("%dx%dx%d" % (_logint(rng, 100, 800), _logint(rng, 8, 96),
                                                             rng.randint(1, 8)) for _ in range(n)))
    nv = rng.choice([1, 1, 2, 3]) if kind in ("objective", "marginals") else 1
    side, mside = _logint(rng, 7, 32), _logint(rng, 7, 32)
    hi = {"laplace": 48, "dropin": 64}.get(kind, 128)
    nt = _logint(rng, 4, hi)
    nt = max(3, min(nt, int(2.7e10 / (nv * side * mside) ** 2.6)))
    case = dict(kind=kind, side=side, mside=mside, nt=nt, nb=rng.randint(1, 8 // nv), obs=_logint(rng, 2000, 60000))
    if kind in ("objective", "marginals"):
        case["nv"] = nv
    if kind == "objective":
        case["grad"] = rng.random() < 0.5
    return case


# ------------------------------------------------------------------------ the inputs
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _blocks(nt, b, a, seed, dev):
    """Diagonally dominant SPD blocks D, L, R, T (float64 tensors)."""
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    s = 1.0 / b ** 0.5

    def normal(*shape):
        return torch.randn(shape, generator=g, device=dev, dtype=F64) * s

    D, L, R, T = normal(nt, b, b), normal(nt - 1, b, b), normal(nt, a, b), normal(a, a)
    D = 0.5 * (D + D.transpose(1, 2))
    T = 0.5 * (T + T.T)
    rows = D.abs().sum(2) - D.diagonal(dim1=1, dim2=2).abs() + R.abs().sum(1)
    rows[1:] += L.abs().sum(2)
    rows[:-1] += L.abs().sum(1)
    D += torch.diag_embed(rows + 1.0)
    T += torch.diag(T.abs().sum(1) - T.diagonal().abs() + R.abs().sum((0, 2)) + 1.0)
    return D.contiguous(), L, R, T.contiguous()


def _rhs(n, nrhs, seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(seed + 1000003)
    return torch.randn((n, nrhs) if nrhs > 1 else (n,), generator=g, device=dev, dtype=F64)


def _shapes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["shapes"].split(",")]


def _spec(case, seed):
    from pyinla_gb300.model import CoregionalSpdeAr1, SeparableSpdeAr1, default_theta
    from pyinla_gb300 import spde
    mesh = spde.unit_square_mesh(case["side"], case["mside"])
    if case["kind"] == "dropin":
        seed = 0     # one data set, as in a run: theta and the right-hand side change from seed to seed
    if case.get("nv", 1) > 1:
        return CoregionalSpdeAr1.synthetic(case["side"], case["nt"], case["nb"], case["nv"], case["obs"], seed,
                                           m_side=case["mside"])
    obs = spde.make_observations(mesh, case["nt"], case["obs"], case["nb"], seed)
    if case["kind"] == "laplace":
        rng = np.random.default_rng(seed + 5)
        obs.z *= 0.1
        obs.y = rng.poisson(np.exp(0.3 * rng.standard_normal(case["obs"]))).astype(np.float64)
    return SeparableSpdeAr1(mesh, case["nt"], case["nb"], obs, default_theta())


def _theta(spec, seed):
    return spec.theta0 + 0.05 * np.random.default_rng(seed + 11).standard_normal(spec.theta0.size)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("plain", "bt", "sweeps"):
        from pyinla_gb300 import algs
        nt, b, a = case["nt"], case["b"], case["a"]
        Q = [x for x in _blocks(nt, b, a, seed, "cuda")][:2 if kind == "bt" else 4]
        rhs = _rhs(nt * b + a, case["nrhs"], seed, "cuda")
        if case.get("host"):
            Q, rhs = [x.cpu().numpy() for x in Q], rhs.cpu().numpy()
        if kind == "sweeps":
            algs.pobtaf(*Q)
        copy = np.empty_like if case.get("host") else torch.empty_like
        return dict(case=case, Q=Q, rhs=rhs, W=[copy(x) for x in Q], x=copy(rhs))
    if kind == "batch":
        from pyinla_gb300.batch import BtaBatch
        shapes = _shapes(case)
        batch = BtaBatch(shapes)
        data = []
        for k, (b, nt, a) in enumerate(shapes):
            data.append(_blocks(nt, b, a, seed * 64 + k, "cuda") + (_rhs(nt * b + a, 1, seed * 64 + k, "cuda"),))
        return dict(case=case, batch=batch, data=data)
    spec = _spec(case, seed)
    theta = _theta(spec, seed)
    if kind == "dropin":
        from pyinla_gb300.solver import GB300SerinvSolver
        _, Qc = spec.sparse_precisions(theta)
        solver = GB300SerinvSolver(diagonal_blocksize=spec.b, n_diag_blocks=spec.nt, arrowhead_blocksize=spec.nb)
        return dict(case=case, solver=solver, Q=Qc, rhs=np.random.default_rng(seed).standard_normal(spec.N))
    if kind == "laplace":
        from pyinla_gb300.laplace import KronLaplaceModel
        return dict(case=case, model=KronLaplaceModel(spec, "poisson"), theta=theta)
    from pyinla_gb300.model import KronGaussianModel
    return dict(case=case, model=KronGaussianModel(spec), theta=theta)


# ------------------------------------------------------------------------- one pass
def _fill(dst, src):
    if isinstance(dst, np.ndarray):
        np.copyto(dst, src)
    else:
        dst.copy_(src)


def run(state):
    from pyinla_gb300 import algs
    case = state["case"]
    kind = case["kind"]
    if kind in ("plain", "bt", "sweeps"):
        _fill(state["x"], state["rhs"])
        if kind == "sweeps":
            algs.pobtas(*state["Q"], state["x"], trans="N")
            algs.pobtas(*state["Q"], state["x"], trans="C")
            return dict(x=state["x"])
        W, x = state["W"], state["x"]
        for w, q in zip(W, state["Q"]):
            _fill(w, q)
        if kind == "bt":
            algs.pobtf(*W)
            logdet = algs.logdet(W[0], sparsity="bt")
            algs.pobts(*W, x, trans="N")
            algs.pobts(*W, x, trans="C")
            algs.pobtsi(*W)
        else:
            algs.pobtaf(*W)
            logdet = algs.logdet(W[0], W[3])
            algs.pobtas(*W, x, trans="N")
            algs.pobtas(*W, x, trans="C")
            if case["selinv"]:
                algs.pobtasi(*W)
        return dict(logdet=logdet, x=x, blocks=W)
    if kind == "batch":
        batch = state["batch"]
        for k, (D, L, R, T, rhs) in enumerate(state["data"]):
            batch.load(k, D, L, R, T, rhs)
        logdets = batch.run()
        return dict(logdet=logdets, x=batch.rhs, D=batch.D, L=batch.L, R=batch.R, T=batch.T)
    if kind == "dropin":
        s = state["solver"]
        s.cholesky(state["Q"], "bta")
        logdet = s.logdet("bta")
        x = s.solve(state["rhs"].copy(), "bta")
        s.selected_inversion("bta")
        S = s._structured_to_spmatrix(state["Q"], "bta")
        return dict(logdet=logdet, x=x, data=S.data, indices=S.indices, indptr=S.indptr)
    model = state["model"]
    if kind == "marginals":
        latent, obs = model.marginal_variances(state["theta"])
        return dict(latent=latent, obs=obs)
    if kind == "laplace":
        model.x_latent = torch.zeros_like(model.x_latent)   # a cold start, as a program's first call
        return dict(f=model.evaluate(state["theta"]), mode=model.x_latent)
    if case["grad"]:
        f, g = model.evaluate(state["theta"], gradient=True)
        return dict(f=f, grad=g, mu=model.mu)
    return dict(f=model.evaluate(state["theta"]), mu=model.mu)


# -------------------------------------------------------------------------- the work
def _flops(nt, b, a, factor=1, selinv=0, solves=0):
    f = nt * b ** 3 / 3 + (nt - 1) * 2 * b ** 3 + (nt - 1) * 2 * a * b * b + nt * (a * b * b + a * a * b) + a ** 3 / 3
    s = (nt - 1) * 17 / 3 * b ** 3 + b ** 3 + nt * 4 * a * b * b
    v = 4 * (nt * b * b / 2 + (nt - 1) * b * b + nt * a * b)
    return factor * f + selinv * s + solves * v


def _bytes(nt, b, a):
    """The blocks of one triangle, once."""
    return 8 * (nt * b * (b + 1) / 2 + (nt - 1) * b * b + nt * a * b + a * (a + 1) / 2)


def work(case):
    kind = case["kind"]
    if kind in ("plain", "bt", "sweeps"):
        nt, b, a, r = case["nt"], case["b"], case["a"], case["nrhs"]
        vec = 16 * r * (nt * b + a)
        if kind == "sweeps":
            return dict(bytes=_bytes(nt, b, a) + vec, flops=_flops(nt, b, a, 0, 0, r))
        selinv = 1 if kind == "bt" else int(case["selinv"])
        return dict(bytes=2 * _bytes(nt, b, a) + vec, flops=_flops(nt, b, a, 1, selinv, r))
    if kind == "batch":
        return dict(bytes=sum(2 * _bytes(nt, b, a) for b, nt, a in _shapes(case)),
                    flops=sum(_flops(nt, b, a, 1, 1, 1) for b, nt, a in _shapes(case)))
    nv = case.get("nv", 1)
    nt, b, a = case["nt"], nv * case["side"] * case["mside"], nv * case["nb"]
    nnz = 8 * (nt * b * (10 * nv + a) + 13 * nv * nv * 3 * b)     # A^T A and the spatial matrices
    if kind == "dropin":
        return dict(bytes=4 * 8 * nt * b * 39, flops=_flops(nt, b, a, 1, 1, 1))
    if kind == "laplace":
        return dict(bytes=nnz, flops=_flops(nt, b, a, 3, 0, 3))   # at least three Newton steps
    if kind == "marginals":
        return dict(bytes=nnz, flops=_flops(nt, b, a, 1, 1, 0))
    return dict(bytes=nnz, flops=_flops(nt, b, a, 1, int(case["grad"]), 1))


# ------------------------------------------------------- the same results in plain torch
def _factor(D, L, R, T):
    """Block Cholesky, top-down; lists of blocks (autograd goes through it)."""
    D, R = list(D), list(R)
    L = list(L)
    for i in range(len(D)):
        D[i] = torch.linalg.cholesky(D[i])
        P = [R[i]] if R[i].shape[0] else []
        if i + 1 < len(D):
            P = [L[i]] + P
        if not P:
            continue
        X = torch.linalg.solve_triangular(D[i], torch.cat(P).T, upper=False).T
        if i + 1 < len(D):
            L[i] = X[: D[i].shape[0]]
            D[i + 1] = D[i + 1] - L[i] @ L[i].T
        if R[i].shape[0]:
            R[i] = X[X.shape[0] - R[i].shape[0]:]
            if i + 1 < len(D):
                R[i + 1] = R[i + 1] - R[i] @ L[i].T
            T = T - R[i] @ R[i].T
    if T.shape[0]:
        T = torch.linalg.cholesky(T)
    return D, L, R, T


def _logdet(D, T):
    return 2.0 * (sum(torch.log(d.diagonal()).sum() for d in D) + torch.log(T.diagonal()).sum())


def _forward(D, L, R, T, v):
    b, nt = D[0].shape[0], len(D)
    v = v.reshape(v.shape[0], -1)
    ys, s, tip = [], v[:b], v[nt * b:]
    for i in range(nt):
        ys.append(torch.linalg.solve_triangular(D[i], s, upper=False))
        if i + 1 < nt:
            s = v[(i + 1) * b:(i + 2) * b] - L[i] @ ys[i]
        tip = tip - R[i] @ ys[i]
    return ys, torch.linalg.solve_triangular(T, tip, upper=False) if T.shape[0] else tip


def _solve(D, L, R, T, v):
    ys, tip = _forward(D, L, R, T, v)
    xt = torch.linalg.solve_triangular(T.T, tip, upper=True) if T.shape[0] else tip
    xs = [None] * len(D)
    for i in reversed(range(len(D))):
        s = ys[i] - R[i].T @ xt
        if i + 1 < len(D):
            s = s - L[i].T @ xs[i + 1]
        xs[i] = torch.linalg.solve_triangular(D[i].T, s, upper=True)
    return torch.cat(xs + [xt]).reshape(v.shape)


def _selinv(D, L, R, T):
    nt, b, a = len(D), D[0].shape[0], T.shape[0]
    eye = torch.eye(b, dtype=F64, device=D[0].device)
    ST = torch.cholesky_inverse(T) if a else T
    SD, SL, SR = [None] * nt, [None] * (nt - 1), [None] * nt
    for i in reversed(range(nt)):
        Finv = torch.linalg.solve_triangular(D[i], eye, upper=False)
        Ri = R[i] @ Finv
        S = Finv.T @ Finv
        SR[i] = -ST @ Ri
        if i + 1 < nt:
            Li = L[i] @ Finv
            SL[i] = -(SD[i + 1] @ Li + SR[i + 1].T @ Ri)
            SR[i] = SR[i] - SR[i + 1] @ Li
            S = S - Li.T @ SL[i]
        S = S - Ri.T @ SR[i]
        SD[i] = 0.5 * (S + S.T)
    return SD, SL, SR, ST


def _stack(xs, like):
    return torch.stack(xs) if len(xs) else like


def _dense(m, dev):
    return torch.from_numpy(m.toarray()).to(dev)


def _ar1(rho, nt):
    """Diagonal and sub-diagonal of the unit-variance AR(1) precision (torch scalars)."""
    s = 1.0 / (1.0 - rho * rho)
    inner = (1.0 + rho * rho) * s
    return torch.stack([s] + [inner] * (nt - 2) + [s]), (-rho * s).expand(nt - 1)


def _variates(spec, case, th):
    """Per variate: scale c, (rho, w) of its prior c T(rho) (x) sum_j w_j S_j, loadings row, tau_y."""
    out = []
    for k in range(spec.nv):
        if spec.nv == 1:
            kap, rt, c, ty = torch.exp(th[0]), torch.exp(th[1]), torch.exp(th[2]), torch.exp(th[3])
            v = torch.ones(1, dtype=F64)
        else:
            kap, rt, ty = (torch.exp(th[3 * k + j]) for j in range(3))
            c = torch.tensor(float(spec.sigma[k]) ** -2.0, dtype=F64)
            v = torch.zeros(spec.nv, dtype=F64)
            v[k] = 1.0
            if k == 1:
                v[0] = -spec.lam["0_1"]
            if k == 2:
                v[0], v[1] = -spec.lam["1_2"], -spec.lam["0_2"]
        out.append((c, torch.exp(-1.0 / rt), torch.stack([kap ** 4, 2.0 * kap ** 2, torch.ones_like(kap)]), v, ty))
    return out


def _gram_blocks(spec, weights, dev):
    """Diagonal blocks, arrow rows and tip of A^T diag(weights) A."""
    A = spec.A.tocsr()
    G = (A.T @ A.multiply(weights[:, None]).tocsr()).tocsr()
    b, nt = spec.b, spec.nt
    D = [_dense(G[t * b:(t + 1) * b, t * b:(t + 1) * b], dev) for t in range(nt)]
    Rall = _dense(G[nt * b:], dev)
    return D, [Rall[:, t * b:(t + 1) * b] for t in range(nt)], Rall[:, nt * b:]


def _prior(spec, case, th, dev):
    """Prior blocks D, L, tip and logdet (without the tip), from theta (a torch vector)."""
    S = [_dense(m, dev) for m in (spec.base_terms if spec.nv > 1 else spec.terms)]
    nt, ns = spec.nt, spec.ns
    D, L, logdet = [0.0] * nt, [0.0] * (nt - 1), 0.0
    for c, rho, w, v, _ in _variates(spec, case, th):
        diag, off = _ar1(rho, nt)
        Qs = sum(w[j].to(dev) * S[j] for j in range(3))
        M = c.to(dev) * torch.kron(torch.outer(v, v).to(dev), Qs)
        D = [D[t] + diag[t].to(dev) * M for t in range(nt)]
        L = [L[t] + off[t].to(dev) * M for t in range(nt - 1)]
        ld = 2.0 * torch.log(torch.linalg.cholesky(Qs).diagonal()).sum().cpu()
        logdet = logdet + nt * ns * torch.log(c) - ns * (nt - 1) * torch.log(1.0 - rho * rho) + nt * ld
    return D, L, spec.tip_prec * torch.eye(spec.nb, dtype=F64, device=dev), logdet


def _log_prior(spec, th):
    return -0.5 * spec.prior_prec * ((th - torch.from_numpy(spec.theta0)) ** 2).sum()


def _conditional(spec, case, th, dev):
    D, L, T, logdet_p = _prior(spec, case, th, dev)
    ov = spec.obs_variates()
    R = [0.0] * spec.nt
    taus = [v[4] for v in _variates(spec, case, th)]
    for k in range(spec.nv):
        GD, GR, GT = _gram_blocks(spec, (ov == k).astype(np.float64), dev)
        t = taus[k].to(dev)
        D = [d + t * g for d, g in zip(D, GD)]
        R = [r + t * g for r, g in zip(R, GR)]
        T = T + t * GT
    return D, L, R, T, logdet_p, taus


def _exact_objective(spec, case, theta, grad, dev):
    th = torch.from_numpy(theta.copy()).requires_grad_(grad)
    D, L, R, T, logdet_p, taus = _conditional(spec, case, th, dev)
    ov, y = spec.obs_variates(), spec.y
    rhs, lik = 0.0, 0.0
    for k in range(spec.nv):
        yk = np.where(ov == k, y, 0.0)
        rhs = rhs + taus[k].to(dev) * torch.from_numpy(spec.A.T @ yk).to(dev)
        lik = lik + 0.5 * int((ov == k).sum()) * torch.log(taus[k]) - 0.5 * taus[k] * float(yk @ yk)
    F = _factor(D, L, R, T)
    ys, tip = _forward(*F, rhs)
    quad = sum((v * v).sum() for v in ys) + (tip * tip).sum()
    f = -(_log_prior(spec, th) + lik + 0.5 * logdet_p) + 0.5 * (_logdet(F[0], F[3]) - quad).cpu()
    out = dict(f=np.float64(f.detach()))
    if grad:
        f.backward()
        out["grad"] = th.grad.numpy()
    with torch.no_grad():
        out["mu"] = _solve(*F, rhs)
    return out


def _exact_laplace(spec, case, theta, dev):
    th = torch.from_numpy(theta.copy())
    PD, PL, PT, logdet_p = _prior(spec, case, th, dev)
    b, nt = spec.b, spec.nt
    A = spec.A.tocsr()
    x = torch.zeros(spec.N, dtype=F64, device=dev)
    dx = torch.zeros_like(x)
    for _ in range(51):
        x = x + dx
        eta = A @ x.cpu().numpy()
        w = np.exp(eta)
        xs = [x[t * b:(t + 1) * b] for t in range(nt)]
        q = [PD[t] @ xs[t] for t in range(nt)]
        for t in range(nt - 1):
            q[t + 1] = q[t + 1] + PL[t] @ xs[t]
            q[t] = q[t] + PL[t].T @ xs[t + 1]
        qpx = torch.cat(q + [PT @ x[nt * b:]])
        GD, GR, GT = _gram_blocks(spec, w, dev)
        F = _factor([p + g for p, g in zip(PD, GD)], PL, GR, PT + GT)
        dx = _solve(*F, torch.from_numpy(A.T @ (spec.y - w)).to(dev) - qpx)
        if float(dx.norm()) < 1e-3:
            break
    lik = float(eta @ spec.y - w.sum())
    f = -(float(_log_prior(spec, th)) + lik + 0.5 * float(logdet_p) - 0.5 * float(x @ qpx)
          - 0.5 * float(_logdet(F[0], F[3])))
    return dict(f=np.float64(f), mode=x)


def _exact_marginals(spec, case, theta, dev):
    D, L, R, T, _, _ = _conditional(spec, case, torch.from_numpy(theta.copy()), dev)
    SD, SL, SR, ST = _selinv(*_factor(D, L, R, T))
    b, nt = spec.b, spec.nt
    latent = torch.cat([s.diagonal() for s in SD] + [ST.diagonal()])
    A = spec.A.tocsr()
    A.sort_indices()
    n, m = A.shape[0], 3 + case["nb"]            # three nodes of one time step, then the fixed effects
    col = torch.from_numpy(A.indices.reshape(n, m).astype(np.int64)).to(dev)
    val = torch.from_numpy(A.data.reshape(n, m)).to(dev)
    t, cf, ca = col[:, 0] // b, col[:, :3] % b, col[:, 3:] - nt * b
    D, R = torch.stack(SD), torch.stack(SR)
    vf, va = val[:, :3], val[:, 3:]
    ff = D[t[:, None, None], cf[:, :, None], cf[:, None, :]]
    af = R[t[:, None, None], ca[:, :, None], cf[:, None, :]]
    aa = ST[ca[:, :, None], ca[:, None, :]]
    obs = (torch.einsum("ni,nij,nj->n", vf, ff, vf) + 2.0 * torch.einsum("ni,nij,nj->n", va, af, vf)
           + torch.einsum("ni,nij,nj->n", va, aa, va))
    return dict(latent=latent.cpu().numpy(), obs=obs.cpu().numpy())


def _exact_dropin(spec, case, theta, seed, dev):
    _, Q = spec.sparse_precisions(theta)          # the input matrix itself
    b, nt = spec.b, spec.nt
    nb = nt * b
    D = [_dense(Q[t * b:(t + 1) * b, t * b:(t + 1) * b], dev) for t in range(nt)]
    L = [_dense(Q[(t + 1) * b:(t + 2) * b, t * b:(t + 1) * b], dev) for t in range(nt - 1)]
    R = [_dense(Q[nb:, t * b:(t + 1) * b], dev) for t in range(nt)]
    F = _factor(D, L, R, _dense(Q[nb:, nb:], dev))
    x = _solve(*F, torch.from_numpy(np.random.default_rng(seed).standard_normal(spec.N)).to(dev))
    SD, SL, SR, ST = _selinv(*F)
    SD, SL, SR = torch.stack(SD), torch.stack(SL), torch.stack(SR)
    Q = Q.tocoo()
    low = Q.row >= Q.col                                  # the result has the lower pattern, mirrored
    r, c = Q.row[low].astype(np.int64), Q.col[low].astype(np.int64)
    off = r > c
    r, c = np.concatenate([r, c[off]]), np.concatenate([c, r[off]])
    order = np.lexsort((r, c))
    r, c = torch.from_numpy(r[order]).to(dev), torch.from_numpy(c[order]).to(dev)
    lo, hi = torch.minimum(r, c), torch.maximum(r, c)     # the lower triangle: row hi, column lo
    data = torch.zeros(r.numel(), dtype=F64, device=dev)
    same, below = (hi < nb) & (hi // b == lo // b), (hi < nb) & (hi // b == lo // b + 1)
    arrow, tip = (hi >= nb) & (lo < nb), lo >= nb
    data[same] = SD[lo[same] // b, hi[same] % b, lo[same] % b]
    data[below] = SL[lo[below] // b, hi[below] % b, lo[below] % b]
    data[arrow] = SR[lo[arrow] // b, hi[arrow] - nb, lo[arrow] % b]
    data[tip] = ST[hi[tip] - nb, lo[tip] - nb]
    return dict(logdet=float(_logdet(F[0], F[3])), x=x.cpu().numpy(), data=data.cpu().numpy(), indices=None, indptr=None)


def exact(case, seed):
    kind, dev = case["kind"], _device()
    if kind in ("plain", "bt", "sweeps", "batch"):
        outs = []
        shapes = _shapes(case) if kind == "batch" else [(case["b"], case["nt"], case["a"])]
        for k, (b, nt, a) in enumerate(shapes):
            s = seed * 64 + k if kind == "batch" else seed
            F = _factor(*_blocks(nt, b, a, s, dev))
            x = _solve(*F, _rhs(nt * b + a, case.get("nrhs", 1), s, dev))
            S = F
            if kind in ("bt", "batch") or case.get("selinv"):
                S = _selinv(*F)
            SD, SL, SR = torch.stack(S[0]), torch.stack(S[1]), torch.stack(S[2])
            outs.append((float(_logdet(F[0], F[3])), x, SD, SL, SR, S[3]))
        if kind == "sweeps":
            return dict(x=outs[0][1])
        if kind == "batch":
            return dict(logdet=np.array([o[0] for o in outs]), x=[o[1] for o in outs], D=[o[2] for o in outs],
                        L=[o[3] for o in outs], R=[o[4] for o in outs], T=[o[5] for o in outs])
        blocks = list(outs[0][2:4 if kind == "bt" else 6])
        x = outs[0][1]
        if case.get("host"):
            blocks, x = [v.cpu().numpy() for v in blocks], x.cpu().numpy()
        return dict(logdet=outs[0][0], x=x, blocks=blocks)
    spec = _spec(case, seed)
    theta = _theta(spec, seed)
    if kind == "dropin":
        return _exact_dropin(spec, case, theta, seed, dev)
    if kind == "laplace":
        return _exact_laplace(spec, case, theta, dev)
    if kind == "marginals":
        return _exact_marginals(spec, case, theta, dev)
    return _exact_objective(spec, case, theta, case["grad"], dev)
