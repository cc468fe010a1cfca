"""The work that users of this library have it do, as timed cases.

Every case goes through the public entry points (include/sddd.h, bound by the
package's Context and Batch): the MPLAPACK-shaped kernels on device memory,
one Newton pass at a given point for each of the problem shapes the workload
generators make, and whole solves, alone, with their gradient and in a batch.

    listed()             the listed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  problem, point and handle, on the GPU
    run(state)           one pass and its outputs
    work(case)           bytes and FP64 operations a pass cannot do without
    exact(case, seed)    the same outputs in plain 64-bit torch
"""
import importlib

import numpy as np
import torch

sddd = importlib.import_module("sdpa-dd_b200")

DD = sddd.DD
# FP64 operations of one dd multiply-add (9 for the product, 11 for the sum).
FP64_PER_TERM = 20.0


def listed():
    return [
        # A product of two small blocks through the MPLAPACK seam: what a
        # program with many small SDP blocks calls most, bound by latency.
        {"name": "gemm_small", "kind": "gemm", "m": 33, "n": 20, "k": 27, "ta": "N", "tb": "N", "alpha": 1.0, "beta": 0.0},
        # The Jordan products of one max-cut-sized block (order 500).
        {"name": "gemm_500", "kind": "gemm", "m": 500, "n": 500, "k": 500, "ta": "N", "tb": "T", "alpha": -1.0, "beta": 1.0},
        # A Schur system of an ordinary problem, factored and solved in the
        # reference's operation order (the library's default), ragged order.
        {"name": "system_plain", "kind": "system", "n": 1327, "nrhs": 2, "slices": 0},
        # A large Schur system with the tensor-core split (16 slices).
        {"name": "system_split", "kind": "system", "n": 5003, "nrhs": 2, "slices": 16},
        # The headline workload's Newton pass: theta of 200 vertices
        # (m = 9951), split form.
        {"name": "newton_theta", "kind": "newton", "problem": "theta", "n": 200, "p": 0.5, "slices": 16, "dinf": True},
        # The same kind of problem at an ordinary size in the default form.
        {"name": "newton_theta_plain", "kind": "newton", "problem": "theta", "n": 71, "p": 0.5, "slices": 0, "dinf": False},
        # Max-cut, n = m = 500: one large block, diagonal constraints.
        {"name": "newton_maxcut", "kind": "newton", "problem": "maxcut", "n": 500, "p": 0.02, "slices": 0, "dinf": True},
        # Control-shaped: blocks 100 and 50, m = 1326 dense constraints.
        {"name": "newton_control", "kind": "newton", "problem": "control", "n": 100, "n2": 50, "m": 1326, "slices": 16, "dinf": True},
        # A chain of 200 blocks of order 20 (m = 5990): the sparse Schur path.
        {"name": "newton_chain", "kind": "newton", "problem": "chain", "n": 20, "blocks": 200, "per": 20, "overlap": 10, "slices": 0, "dinf": True},
        # A whole solve of a small max-cut problem to relative gap 1e-25.
        {"name": "solve_maxcut", "kind": "solve", "problem": "maxcut", "n": 100, "p": 0.1, "slices": 0, "grad": False},
        # A whole solve and its gradient with weights on every output (the
        # layer of a differentiable program).
        {"name": "solve_grad", "kind": "solve", "problem": "control", "n": 20, "n2": 10, "m": 150, "slices": 0, "grad": True},
        # A batch of independent small problems, each with d(c.x)/dc.
        {"name": "batch", "kind": "batch", "count": 16, "nmin": 10, "nmax": 80},
    ]


def _log(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["gemm", "system", "system", "newton", "newton", "newton", "newton", "solve", "batch"])
    if kind == "gemm":
        return {"kind": "gemm", "m": _log(rng, 5, 600), "n": _log(rng, 5, 600), "k": _log(rng, 5, 600), "ta": rng.choice("NT"), "tb": rng.choice("NT"),
                "alpha": rng.choice([1.0, -1.0, 0.75]), "beta": rng.choice([0.0, 1.0, 0.5])}
    if kind == "system":
        slices = rng.choice([0, 16])
        return {"kind": "system", "n": _log(rng, 20, 5000 if slices else 2000), "nrhs": rng.choice([1, 2, 3]), "slices": slices}
    if kind == "newton":
        problem = rng.choice(["theta", "theta", "maxcut", "control", "chain"])
        case = {"kind": "newton", "problem": problem, "slices": rng.choice([0, 16]), "dinf": rng.choice([False, True])}
        if problem == "theta":
            case |= {"n": _log(rng, 15, 180 if case["slices"] else 100), "p": round(rng.uniform(0.3, 0.5), 3)}
        elif problem == "maxcut":
            n = _log(rng, 15, 500)
            case |= {"n": n, "p": round(min(0.5, 10.0 / n), 4)}
        elif problem == "control":
            n, n2 = _log(rng, 8, 90), _log(rng, 4, 45)
            room = (n * (n + 1) + n2 * (n2 + 1)) // 2
            case |= {"n": n, "n2": n2, "m": max(4, min(1200, int(room * rng.uniform(0.2, 0.6))))}
        else:
            case |= {"n": rng.randint(5, 24), "blocks": _log(rng, 12, 180), "per": rng.randint(4, 20), "overlap": rng.randint(1, 6), "slices": 0}
        return case
    if kind == "solve":
        if rng.random() < 0.5:
            n = _log(rng, 15, 160)
            return {"kind": "solve", "problem": "maxcut", "n": n, "p": round(min(0.5, 10.0 / n), 4), "slices": rng.choice([0, 16]), "grad": False}
        n, n2 = rng.randint(8, 24), rng.randint(4, 12)
        room = (n * (n + 1) + n2 * (n2 + 1)) // 2
        return {"kind": "solve", "problem": "control", "n": n, "n2": n2, "m": int(room * rng.uniform(0.3, 0.6)), "slices": 0, "grad": True}
    return {"kind": "batch", "count": rng.randint(4, 16), "nmin": rng.randint(10, 16), "nmax": rng.randint(30, 70)}


# ------------------------------------------------------------------ inputs
def _dd(hi, lo=None):
    out = np.zeros(np.shape(hi), DD)
    out["hi"] = hi
    if lo is not None:
        out["lo"] = lo
    return out


def _lo(rng, hi):
    """Low parts that use all of a dd's digits."""
    return np.asarray(hi) * rng.uniform(-1.0, 1.0, np.shape(hi)) * 2.0 ** -54


class _Problem:
    """An SDP in the library's entry form: m, sizes, c, and entries
    (constraint k = 0..m with 0 for F_0, block, row <= column, value)."""

    def __init__(self, m, sizes):
        self.m, self.sizes, self.c = m, list(sizes), np.zeros(m)
        self.parts = []

    def add(self, k, blk, i, j, v):
        n = np.broadcast(k, blk, i, j, v).shape
        types = (np.int16, np.int32, np.int32, np.int32, np.float64)
        self.parts.append([np.broadcast_to(np.asarray(a, t), n).ravel() for a, t in zip((k, blk, i, j, v), types)])

    def done(self):
        """The entries by constraint, each constraint's in the order added."""
        cols = [np.concatenate([p[t] for p in self.parts]) for t in range(5)]
        order = np.argsort(cols[0], kind="stable")
        self.k, self.blk, self.i, self.j, self.v = (a[order] for a in cols)
        self.parts = []
        return self

    def args(self):
        return (self.m, self.sizes, _dd(self.c), self.k, self.blk + 1, self.i + 1, self.j + 1, _dd(self.v))


def _theta(rng, case):
    n = case["n"]
    iu, ju = np.triu_indices(n, 1)
    keep = np.sort(rng.permutation(len(iu))[:int(case["p"] * len(iu))])
    eu, ev = iu[keep], ju[keep]
    P = _Problem(1 + len(eu), [n])
    P.c[0] = 1.0
    du, dv = np.triu_indices(n)
    P.add(0, 0, du, dv, 1.0)
    P.add(1, 0, np.arange(n), np.arange(n), 1.0)
    P.add(2 + np.arange(len(eu)), 0, eu, ev, 1.0)
    return P.done()


def _maxcut(rng, case):
    n = case["n"]
    A = np.triu(rng.random((n, n)) < case["p"], 1)
    w = np.where(A, 0.5 + rng.random((n, n)), 0.0)
    w = w + w.T
    L = (np.diag(w.sum(axis=1)) - w) / 4.0
    P = _Problem(n, [n])
    P.c[:] = 1.0
    i, j = np.nonzero(np.triu(L))
    P.add(0, 0, i, j, L[i, j])
    P.add(1 + np.arange(n), 0, np.arange(n), np.arange(n), 1.0)
    return P.done()


def _dense_blocks(rng, P, blk, ks, x0, n):
    """Constraints ks on a block: dense N(0,1)/sqrt(n), symmetric; F_0 so
    that x0 is strictly feasible; c so that Y = I is."""
    A = rng.standard_normal((len(ks), n, n)) / np.sqrt(n)
    A = 0.5 * (A + A.transpose(0, 2, 1))
    G = rng.standard_normal((n, n))
    F0 = np.tensordot(x0[ks], A, axes=1) - (np.eye(n) + G @ G.T / n)
    iu, ju = np.triu_indices(n)
    P.c[ks] += np.trace(A, axis1=1, axis2=2)
    P.add(0, blk, iu, ju, F0[iu, ju])
    P.add(1 + np.asarray(ks)[:, None], blk, iu[None], ju[None], A[:, iu, ju])


def _control(rng, case):
    sizes = [case["n"], case["n2"]]
    P = _Problem(case["m"], sizes)
    x0 = rng.standard_normal(P.m)
    for b, n in enumerate(sizes):
        _dense_blocks(rng, P, b, np.arange(P.m), x0, n)
    return P.done()


def _chain(rng, case):
    nb, n, per, ov = case["blocks"], case["n"], case["per"], case["overlap"]
    touch = []
    for b in range(nb):
        touch += [[b]] * per
        if b + 1 < nb:
            touch += [[b, b + 1]] * ov
    perm = rng.permutation(len(touch))
    on = [[] for _ in range(nb)]
    for t, bs in enumerate(touch):
        for b in bs:
            on[b].append(perm[t])
    P = _Problem(len(touch), [n] * nb)
    x0 = rng.standard_normal(P.m)
    for b in range(nb):
        _dense_blocks(rng, P, b, np.sort(np.array(on[b])), x0, n)
    return P.done()


_MAKE = {"theta": _theta, "maxcut": _maxcut, "control": _control, "chain": _chain}


def _point(rng, sizes, m):
    """An interior point on the way to a solution: X and Z nearly commuting,
    eigenvalues over three decades, X Z near mu I; y ~ N(0,1)."""
    X, Z = [], []
    for n in sizes:
        Q = np.linalg.qr(rng.standard_normal((n, n)))[0]
        lam = 10.0 ** rng.uniform(-1.5, 1.5, n)
        lz = 0.01 / lam * np.exp(0.3 * rng.standard_normal(n))
        for out, l in ((X, lam), (Z, lz)):
            M = (Q * l) @ Q.T
            M = 0.5 * (M + M.T)
            lo = _lo(rng, M)
            lo = np.triu(lo) + np.triu(lo, 1).T
            out.append((M, lo))
    flat = lambda S: _dd(np.concatenate([a.ravel() for a, _ in S]), np.concatenate([b.ravel() for _, b in S]))  # noqa: E731
    y = rng.standard_normal(m)
    return flat(X), _dd(y, _lo(rng, y)), flat(Z)


class _Handle:
    """Closes a context or batch with the state that holds it."""

    def __init__(self, h):
        self.h = h

    def __del__(self):
        try:
            self.h.close()
        except Exception:
            pass


def _gpu(a):
    """A dd array as an n x 2 device tensor."""
    return torch.from_numpy(np.ascontiguousarray(a).view(np.float64).reshape(-1, 2)).cuda()


def _system(case, seed):
    """A symmetric positive definite dd matrix (column-major, condition about
    1e3) and right-hand sides."""
    n = case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    G = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    A = torch.zeros(n, n, 2, dtype=torch.float64, device="cuda")
    A[:, :, 0] = G @ G.T / n + 0.01 * torch.eye(n, dtype=torch.float64, device="cuda")
    A[:, :, 0] = 0.5 * (A[:, :, 0] + A[:, :, 0].T)
    u = (torch.rand(n, n, dtype=torch.float64, device="cuda", generator=g) - 0.5) * 2.0 ** -53
    A[:, :, 1] = A[:, :, 0] * torch.triu(u) + (A[:, :, 0] * torch.triu(u, 1)).T
    b = torch.randn(case["nrhs"], n, dtype=torch.float64, device="cuda", generator=g)
    B = torch.stack([b, b * 2.0 ** -55], dim=2).contiguous()
    return A, B


def _gemm(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def mat(rows, cols):  # column-major: cols x rows x 2
        hi = torch.randn(cols, rows, dtype=torch.float64, device="cuda", generator=g)
        lo = hi * (torch.rand(cols, rows, dtype=torch.float64, device="cuda", generator=g) - 0.5) * 2.0 ** -53
        return torch.stack([hi, lo], dim=2).contiguous()

    m, n, k = case["m"], case["n"], case["k"]
    A = mat(m, k) if case["ta"] == "N" else mat(k, m)
    B = mat(k, n) if case["tb"] == "N" else mat(n, k)
    return A, B, mat(m, n)


def _batch_problems(case, rng):
    out = []
    shapes = np.random.default_rng([case["count"], case["nmin"], case["nmax"]])  # the sizes belong to the case, the data to the seed
    for _ in range(case["count"]):
        n = int(shapes.integers(case["nmin"], case["nmax"] + 1))
        room = n * (n + 1) // 2
        m = int(min(200, max(4, room * shapes.uniform(0.2, 0.5))))
        P = _Problem(m, [n])
        _dense_blocks(rng, P, 0, np.arange(m), rng.standard_normal(m), n)
        out.append(P.done())
    return out


def _param(eps):
    p = sddd.param()
    p.maxIteration = 200
    p.epsilonStar = p.epsilonDash = eps
    return p


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = {"case": case}
    if kind == "batch":
        B = sddd.Batch()
        s["handle"], s["batch"], s["param"] = _Handle(B), B, _param(1e-15)
        for P in _batch_problems(case, rng):
            B.add(*P.args())
        return s
    ctx = sddd.Context()
    s["handle"], s["ctx"] = _Handle(ctx), ctx
    if kind in ("gemm", "system"):
        s["stream"] = torch.cuda.ExternalStream(ctx.L.sddd_stream(ctx.h))
        if kind == "gemm":
            s["A"], s["B"], s["C0"] = _gemm(case, seed)
            s["C"] = torch.empty_like(s["C0"])
        else:
            ctx.call("sddd_set_tc_split", case["slices"])
            s["A0"], s["B0"] = _system(case, seed)
            s["A"], s["B"] = torch.empty_like(s["A0"]), torch.empty_like(s["B0"])
        torch.cuda.synchronize()
        return s
    ctx.call("sddd_set_tc_split", case["slices"])
    P = _MAKE[case["problem"]](rng, case)
    ctx.upload(*P.args())
    if kind == "newton":
        s["X"], s["y"], s["Z"] = _point(rng, P.sizes, P.m)
    else:
        s["param"] = _param(1e-25 if case["problem"] == "maxcut" else 1e-20)
        if case["grad"]:
            sym = [rng.standard_normal((n, n)) for n in P.sizes]
            sym = np.concatenate([(0.5 * (a + a.T)).ravel() for a in sym])
            s["g"] = (_dd(rng.standard_normal(P.m)), _dd(sym), _dd(-0.5 * sym))
    return s


# -------------------------------------------------------------------- runs
def _arr(a):
    return a.view(np.float64).reshape(-1, 2)


def _run_gemm(s):
    c, ctx = s["case"], s["ctx"]
    A, B, C = s["A"], s["B"], s["C"]
    with torch.cuda.stream(s["stream"]):
        C.copy_(s["C0"])
    ctx.call("sddd_Rgemm", c["ta"].encode(), c["tb"].encode(), c["m"], c["n"], c["k"], sddd.SdddDD(c["alpha"], 0.0), A.data_ptr(), A.shape[1], B.data_ptr(),
             B.shape[1], sddd.SdddDD(c["beta"], 0.0), C.data_ptr(), c["m"])
    return {"hi": C[:, :, 0], "lo": C[:, :, 1]}


def _run_system(s):
    c, ctx = s["case"], s["ctx"]
    A, B, n = s["A"], s["B"], c["n"]
    with torch.cuda.stream(s["stream"]):
        A.copy_(s["A0"])
        B.copy_(s["B0"])
    info = ctx.call("sddd_Rpotrf", b"L", n, A.data_ptr(), n)
    ctx.call("sddd_Rpotrs", b"L", n, c["nrhs"], A.data_ptr(), n, B.data_ptr(), n)
    return {"info": info, "A_hi": A[:, :, 0], "A_lo": A[:, :, 1], "x_hi": B[:, :, 0], "x_lo": B[:, :, 1]}


BETA_MU = 0.003, 0.001


def _run_newton(s):
    ctx, dinf = s["ctx"], int(s["case"]["dinf"])
    if ctx.set_point(s["X"], s["y"], s["Z"]) != 0:
        raise RuntimeError("the point is not positive definite")
    norm_p, norm_d = sddd.SdddDD(), sddd.SdddDD()
    ctx.call("sddd_residuals", norm_p, norm_d)
    ctx.call("sddd_newton_rhs", 0, sddd.SdddDD(BETA_MU[0], 0.0), dinf)
    ctx.call("sddd_schur_build")
    if ctx.call("sddd_schur_factor") != 0:
        raise RuntimeError("the Schur matrix is not positive definite")
    ctx.call("sddd_solve_dy")
    ctx.call("sddd_make_dz_dx", dinf)
    pred = ctx.get("Dy")
    ctx.call("sddd_newton_rhs", 1, sddd.SdddDD(BETA_MU[1], 0.0), dinf)
    ctx.call("sddd_solve_dy")
    ctx.call("sddd_make_dz_dx", dinf)
    eig_x = ctx.dd_scalar("sddd_min_eig", 0)
    eig_z = ctx.dd_scalar("sddd_min_eig", 1)
    return {"norms": np.array([norm_p.hi, norm_d.hi]), "Dy_predictor": _arr(pred), "Dx": _arr(ctx.get("Dx")), "Dy": _arr(ctx.get("Dy")),
            "Dz": _arr(ctx.get("Dz")), "eig": np.array([eig_x, eig_z])}


def _run_solve(s):
    ctx = s["ctx"]
    r = ctx.solve(s["param"])
    out = {"objective": np.array([r.objValPrimal.hi, r.objValDual.hi]), "X": _arr(ctx.get("X")), "y": _arr(ctx.get("y")), "Z": _arr(ctx.get("Z"))}
    if "g" in s:
        grad_c, grad_F0 = ctx.adjoint(*s["g"], g_obj=(1.0, 0.0))
        out["grad_c"], out["grad_F0"] = _arr(grad_c), _arr(grad_F0)
    return out


def _run_batch(s):
    B = s["batch"]
    res = B.solve(s["param"], with_grad=True)
    pts = [B.point(i) for i in range(len(res))]
    cat = lambda t: _arr(np.concatenate([p[t] for p in pts]))  # noqa: E731
    return {"objective": np.array([[r.objValPrimal.hi, r.objValDual.hi] for r in res]), "X": cat(0), "y": cat(1), "Z": cat(2),
            "grad_c": _arr(np.concatenate([B.grad_c(i) for i in range(len(res))]))}


_RUN = {"gemm": _run_gemm, "system": _run_system, "newton": _run_newton, "solve": _run_solve, "batch": _run_batch}


def run(state):
    return _RUN[state["case"]["kind"]](state)


# -------------------------------------------------------------------- work
def _newton_work(case):
    """dd multiply-adds and bytes of one Newton pass: data, point and
    direction once, the Schur matrix written and read once."""
    prob, n = case["problem"], float(case["n"])
    if prob == "theta":
        m, sizes = 1.0 + case["p"] * n * (n - 1) / 2, [n]
        nnz, schur = m + n * n / 2 + n, 4.0 * m * m / 2  # an edge pair: two off-diagonal entries each
    elif prob == "maxcut":
        m, sizes = n, [n]
        nnz, schur = n + case["p"] * n * n / 2 + n, m * m / 2
    elif prob == "control":
        m, sizes = float(case["m"]), [n, float(case["n2"])]
        nnz = (m + 1) * sum(k * (k + 1) / 2 for k in sizes)
        schur = sum(m * 2 * k ** 3 + m * m / 2 * k * k for k in sizes)
    else:
        c = case["per"] + 2.0 * case["overlap"]  # constraints on a block
        m, sizes = case["blocks"] * (case["per"] + case["overlap"]) - case["overlap"], [n] * case["blocks"]
        nnz = case["blocks"] * (c + 1) * n * (n + 1) / 2
        schur = case["blocks"] * (c * 2 * n ** 3 + c * c / 2 * n * n)
    if prob == "chain":
        chol, entries = case["blocks"] * c ** 3 / 6, case["blocks"] * c * c / 2
    else:
        chol, entries = m ** 3 / 6, m * m / 2
    space = sum(k * k for k in sizes)
    cube = sum(k ** 3 for k in sizes)
    terms = schur + chol + 4 * entries + 10 * cube
    return 16 * (nnz + 5 * space + 4 * m + 2 * entries), FP64_PER_TERM * terms


def work(case):
    kind = case["kind"]
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        c = 2 if case["beta"] != 0.0 else 1
        return {"bytes": 16.0 * (m * k + k * n + c * m * n), "flops": FP64_PER_TERM * m * n * k}
    if kind == "system":
        n, r = float(case["n"]), case["nrhs"]
        return {"bytes": 16.0 * (n * n + 2 * n * r), "flops": FP64_PER_TERM * (n ** 3 / 6 + r * n * n)}
    if kind == "newton":
        b, f = _newton_work(case)
        return {"bytes": b, "flops": f}
    # a solve: the passes a primal-dual method needs to its gap (about 35
    # to 1e-25, 20 to 1e-15), each one Newton pass
    if kind == "solve":
        b, f = _newton_work(case)
        return {"bytes": 35 * b, "flops": 35 * f}
    n = 0.5 * (case["nmin"] + case["nmax"])
    b, f = _newton_work({"problem": "control", "n": n, "n2": 0, "m": min(200, 0.35 * n * (n + 1) / 2)})
    return {"bytes": 20 * case["count"] * b, "flops": 20 * case["count"] * f}


# ------------------------------------------------------------------- exact
def _exact_gemm(case, seed):
    A, B, C = (t[:, :, 0].T for t in _gemm(case, seed))  # back to rows x columns
    if case["ta"] == "T":
        A = A.T
    if case["tb"] == "T":
        B = B.T
    return {"hi": (case["alpha"] * (A @ B) + case["beta"] * C).T.contiguous(), "lo": None}


def _exact_system(case, seed):
    A, B = _system(case, seed)
    A, b = A[:, :, 0], B[:, :, 0]
    L = torch.linalg.cholesky(A)
    # column-major storage: the factor's lower triangle, the input above it
    out = torch.triu(L.T) + torch.tril(A, -1)
    return {"info": 0, "A_hi": out, "A_lo": None, "x_hi": torch.cholesky_solve(b.T, L).T.contiguous(), "x_lo": None}


def _exact_newton(case, seed):
    rng = np.random.default_rng(seed)
    P = _MAKE[case["problem"]](rng, case)
    X, y, Z = _point(rng, P.sizes, P.m)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
    m, b, yt = P.m, t(P.c), t(y["hi"])
    blocks, off = [], 0
    for l, n in enumerate(P.sizes):
        e = np.nonzero(P.blk == l)[0]
        ks = np.unique(P.k[e])
        M = torch.zeros(len(ks), n, n, dtype=torch.float64, device=dev)
        pos, i, j, v = t(np.searchsorted(ks, P.k[e])), t(P.i[e].astype(np.int64)), t(P.j[e].astype(np.int64)), t(P.v[e])
        M[pos, i, j] = v
        M[pos, j, i] = v
        has0 = ks[0] == 0
        C = -M[0] if has0 else torch.zeros(n, n, dtype=torch.float64, device=dev)
        A, ids = (M[1:], ks[1:] - 1) if has0 else (M, ks - 1)
        Xl, Zl = (t(s["hi"][off:off + n * n].reshape(n, n)) for s in (X, Z))
        off += n * n
        blocks.append((A, t(ids.astype(np.int64)), C, Xl, Zl, torch.linalg.inv(Zl)))
    dot_A = lambda S: torch.zeros(m, dtype=torch.float64, device=dev).index_add_(0, torch.cat([k[1] for k in blocks]), torch.cat(  # noqa: E731
        [k[0].flatten(1) @ s.flatten() for k, s in zip(blocks, S)]))
    sum_A = lambda v: [torch.tensordot(v[k[1]], k[0], dims=1) for k in blocks]  # noqa: E731
    rp = b - dot_A([k[3] for k in blocks])
    rd = [k[2] - k[4] - s for k, s in zip(blocks, sum_A(yt))]
    B = torch.zeros(m, m, dtype=torch.float64, device=dev)
    for A, ids, _, Xl, _, Zi in blocks:
        B[ids[:, None], ids[None, :]] += A.flatten(1) @ (Xl @ A @ Zi).flatten(1).T
    L = torch.linalg.cholesky(0.5 * (B + B.T))
    del B

    def step(beta_mu, extra):
        R = [beta_mu * k[5] - k[3] - e for k, e in zip(blocks, extra)]
        W = [r - k[3] @ d @ k[5] for r, k, d in zip(R, blocks, rd)] if case["dinf"] else R
        dy = torch.cholesky_solve((rp - dot_A(W))[:, None], L)[:, 0]
        dz = [(d if case["dinf"] else 0) - s for d, s in zip(rd, sum_A(dy))]
        dx = [r - k[3] @ d @ k[5] for r, k, d in zip(R, blocks, dz)]
        return dy, [0.5 * (a + a.T) for a in dx], dz

    dy0, dx, dz = step(BETA_MU[0], [0.0] * len(blocks))
    dy, dx, dz = step(BETA_MU[1], [a @ c @ k[5] for a, c, k in zip(dx, dz, blocks)])

    def flat(v):  # n x 2 as the library's, the low parts below 64 bits
        v = torch.cat([x.flatten() for x in v])
        return torch.stack([v, torch.zeros_like(v)], dim=1)

    norms = torch.stack([rp.abs().max(), torch.stack([d.abs().max() for d in rd]).max()])
    # the step-length eigenvalue is the reference's Lanczos bound, which
    # stops at a relative accuracy of its own: no value to compare with
    return {"norms": norms, "Dy_predictor": flat([dy0]), "Dx": flat(dx), "Dy": flat([dy]), "Dz": flat(dz), "eig": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        return _exact_gemm(case, seed)
    if kind == "system":
        return _exact_system(case, seed)
    if kind == "newton":
        return _exact_newton(case, seed)
    # a solve's final point is a limit, not a formula in 64 bits
    return None
