"""The measured workloads of the platform.

Each listed case is a call a program makes in earnest: whole solves of the
configurations this repository is built for (2-D and 3-D Q1 systems, FP64 and
mixed precision, Jacobi, multicolour SGS and ILU preconditioners), the solve
server's batch, a host-driven Krylov loop over the vector and matrix
operations, a multigrid level step, and the product of an unstructured CSR.
``draw`` gives further cases of the same kinds over the whole size ranges.
"""
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

DEV = "cuda"
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "hiflow3_b200"
    if name not in sys.modules:
        d = os.path.join(ROOT, "hiflow3_2.0_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


_pf = None


def _platform():
    """The program's one platform (init_platform once per process)."""
    global _pf
    if _pf is None:
        _pf = _package().Platform(0)
    return _pf


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # a small time step's system: every iteration is a few microseconds of
        # work, so launches and reductions are all there is
        dict(name="pcg_2d_33", kind="pcg", dim=2, N=33),
        # the 2-D Poisson configuration (66,049 dofs), resident in L2
        dict(name="pcg_2d_256", kind="pcg", dim=2, N=256),
        # FP64 Jacobi-CG on a 3-D heterogeneous system, rows ragged against 32
        dict(name="pcg_3d_100", kind="pcg", dim=3, N=100),
        # the headline: FP32 CG inside FP64 defect correction, 2.1 M dofs
        dict(name="mpir_3d_128", kind="mpir", dim=3, N=128),
        # CG with the 8-colour symmetric Gauss-Seidel preconditioner
        dict(name="mcsgs_3d_96", kind="mcsgs", dim=3, N=96),
        # convection-diffusion, GMRES(30) + level-scheduled ILU(0), FP64
        dict(name="gmres_ilu0_512", kind="gmres", N=512, p=0, mixed=False),
        # the same in mixed precision, at an ordinary size
        dict(name="gmres_ilu0_mixed_300", kind="gmres", N=300, p=0, mixed=True),
        # ILU(1): longer rows, more levels, fewer iterations
        dict(name="gmres_ilu1_200", kind="gmres", N=200, p=1, mixed=False),
        # one product of an unstructured FE-like operator (ragged rows)
        dict(name="spmv_csr_600001", kind="spmv", n=600001, mean=21, f32=False),
        # the host application's own CG over VectorMult, Dot, Axpy, ScaleAdd
        dict(name="lmp_cg_2d_181", kind="lmp_cg", dim=2, N=181, its=30),
        # a multigrid level step: residual, restriction, prolongation
        dict(name="gmg_3d_64", kind="gmg", dim=3, N=64),
        # the solve server on a batch of the mixed request stream
        dict(name="serve_40", kind="serve", count=40, nmax=512, mmax=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pcg", "pcg", "mpir", "mcsgs", "gmres", "gmres", "spmv", "lmp_cg", "gmg", "serve"])
    if kind == "pcg":
        dim = rng.choice([2, 3])
        return dict(kind=kind, dim=dim, N=_log_int(rng, 24, 512) if dim == 2 else _log_int(rng, 12, 100))
    if kind == "mpir":
        dim = rng.choice([2, 3])
        return dict(kind=kind, dim=dim, N=_log_int(rng, 48, 512) if dim == 2 else _log_int(rng, 24, 120))
    if kind == "mcsgs":
        dim = rng.choice([2, 3])
        return dict(kind=kind, dim=dim, N=_log_int(rng, 48, 400) if dim == 2 else _log_int(rng, 16, 96))
    if kind == "gmres":
        p = rng.choice([0, 0, 1])
        return dict(kind=kind, N=_log_int(rng, 48, 500 if p == 0 else 240), p=p, mixed=rng.choice([False, True]))
    if kind == "spmv":
        return dict(kind=kind, n=_log_int(rng, 20000, 600000), mean=rng.randint(5, 30), f32=rng.choice([False, True]))
    if kind == "lmp_cg":
        dim = rng.choice([2, 3])
        return dict(kind=kind, dim=dim, N=_log_int(rng, 32, 500) if dim == 2 else _log_int(rng, 12, 64),
                    its=rng.randint(10, 30))
    if kind == "gmg":
        dim = rng.choice([2, 3])
        return dict(kind=kind, dim=dim, N=2 * _log_int(rng, 24, 200) if dim == 2 else 2 * _log_int(rng, 8, 32))
    return dict(kind=kind, count=rng.randint(8, 40), nmax=rng.randint(64, 512), mmax=rng.randint(20, 64))


# ------------------------------------------------------------------ inputs

def _field(N, dim, sigma, ell, seed):
    """Log-normal coefficient exp(g) on the N^dim cells (x fastest): g a Gaussian
    field of squared-exponential covariance by randomised spectral sampling
    (128 cosine modes of wave vectors drawn from the covariance's spectrum)."""
    rng = np.random.default_rng(seed)
    m = 128
    k = rng.standard_normal((dim, m)) / ell
    phase = rng.uniform(0, 2 * np.pi, m)
    x = torch.from_numpy((np.arange(N) + 0.5) / N).to(DEV)
    e = [torch.exp(1j * torch.outer(x, torch.from_numpy(k[d]).to(DEV))) for d in range(dim)]
    e[0] = e[0] * torch.exp(1j * torch.from_numpy(phase).to(DEV))
    outer = e[1] if dim == 2 else (e[2][:, None, :] * e[1][None, :, :]).reshape(N * N, m)
    g = (outer @ e[0].T).real * (sigma * math.sqrt(2.0 / m))
    return torch.exp(g).reshape(-1).cpu().numpy()


def _interior(dim, N):
    axis = (np.arange(N + 1) > 0) & (np.arange(N + 1) < N)
    m = axis
    for _ in range(dim - 1):
        m = np.logical_and.outer(axis, m)
    return m.reshape(-1)


def _rhs(dim, N, seed):
    """Uniform [-1, 1) on the interior dofs, 0 on the Dirichlet ones."""
    b = np.random.default_rng(seed + 7).uniform(-1.0, 1.0, (N + 1) ** dim)
    b[~_interior(dim, N)] = 0.0
    return b


def _sigma(case):
    return 1.0 if case["dim"] == 3 else 0.5


def _csr_unstructured(case, seed):
    """An FE-like operator in a bandwidth-reduced numbering: ragged rows, columns
    scattered about the diagonal, a few far couplings."""
    rng = np.random.default_rng(seed)
    n, mean = case["n"], case["mean"]
    length = rng.integers(max(1, mean // 2), mean + mean // 2 + 1, n)
    row = np.zeros(n + 1, np.int64)
    np.cumsum(length, out=row[1:])
    i = np.repeat(np.arange(n), length)
    off = np.rint(rng.standard_normal(i.size) * 400.0).astype(np.int64)
    far = rng.random(i.size) < 0.02
    col = np.where(far, rng.integers(0, n, i.size), np.clip(i + off, 0, n - 1))
    i, col = np.divmod(np.unique(i * n + col), n)
    np.cumsum(np.bincount(i, minlength=n), out=row[1:])
    return row.astype(np.int32), col.astype(np.int32), rng.uniform(-1.0, 1.0, i.size), rng.uniform(-1.0, 1.0, n)


def _interp(dim, Nc):
    """Multilinear interpolation from (Nc+1)^dim coarse to (2 Nc+1)^dim fine nodes, as COO."""
    f = np.arange(2 * Nc + 1)
    r1 = np.concatenate([f[::2], f[1::2], f[1::2]])
    c1 = np.concatenate([f[::2] // 2, f[1::2] // 2, f[1::2] // 2 + 1])
    v1 = np.concatenate([np.ones(Nc + 1), np.full(2 * Nc, 0.5)])
    r, c, v = r1, c1, v1
    for d in range(1, dim):
        r = (r1[:, None] * (2 * Nc + 1) ** d + r[None, :]).reshape(-1)
        c = (c1[:, None] * (Nc + 1) ** d + c[None, :]).reshape(-1)
        v = (v1[:, None] * v[None, :]).reshape(-1)
    return r, c, v


def _to_csr(r, c, v, n):
    o = np.lexsort((c, r))
    row = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=n), out=row[1:])
    return row, c[o].astype(np.int32), v[o]


def _requests(case, seed):
    """The request mix of the serving stream: 80 % 2-D systems with log-normal
    coefficients, 20 % 3-D ones, half of them in mixed precision (the sizes
    are the case's, the values the seed's)."""
    rng, values = np.random.default_rng(case["count"] + case["nmax"]), np.random.default_rng(seed)
    out = []
    for k in range(case["count"]):
        dim = 3 if k % 5 == 4 else 2
        N = int(rng.integers(32, case["nmax"] + 1)) if dim == 2 else int(rng.integers(16, case["mmax"] + 1))
        out.append(dict(dim=dim, N=N, mixed=bool(rng.random() < 0.5), seed=int(values.integers(1 << 30))))
    return out


# ------------------------------------------------------------------ prepare / run

GMRES_NU, GMRES_BETA = 1e-3, (1.0, 0.5)


class _Served:
    """The program's server and its request batch."""

    def __init__(self, case, seed):
        b200 = _package()
        srv = importlib.import_module("hiflow3_b200.serving")
        self.server = srv.Server()
        self.batch = []
        for q in _requests(case, seed):
            kc = _field(q["N"], 2, 0.5, 0.1, q["seed"]) if q["dim"] == 2 else None
            self.batch.append(dict(q1=dict(dim=q["dim"], N=q["N"], kcell=kc), b=_rhs(q["dim"], q["N"], q["seed"]),
                                   precision=b200.SERVE_MIXED if q["mixed"] else b200.SERVE_F64,
                                   ctl=(100000, 0.0, 1e-11, 1e6)))

    def run(self):
        ids = [self.server.submit(**a) for a in self.batch]
        return [self.server.wait(i)["x"] for i in ids]


def prepare(case, seed):
    b200, kind = _package(), case["kind"]
    if kind == "serve":
        return dict(case=case, served=_Served(case, seed))
    pf = _platform()
    s = dict(case=case, pf=pf)
    if kind == "spmv":
        dt = b200.F32 if case["f32"] else b200.F64
        row, col, val, x = _csr_unstructured(case, seed)
        s.update(A=b200.CSR_lMatrix.from_csr(pf, row, col, val, dtype=dt), x=pf.vector(x, dt),
                 y=pf.vector(case["n"], dt))
        return s
    if kind == "gmres":
        N = case["N"]
        row, col, val = b200.q1_assemble(2, N, 1, None, GMRES_NU, GMRES_BETA)
        args = (pf, row, col, val)
        make = (lambda dt: b200.Preconditioner.ILU0(*args, dtype=dt)) if case["p"] == 0 else \
            (lambda dt: b200.Preconditioner.ILUp(*args, case["p"], mode=b200.PRECOND_ILU0_LS, dtype=dt))
        P = make(b200.F64)
        if case["mixed"]:
            P32 = make(b200.F32)
            solver = b200.MPIR(pf)
            solver.SetupOperator(P.A_perm)
            solver.SetupLowPrecisionOperator(P32.A_perm)
            solver.SetupInnerGMRES(30, P32)
            solver.InitControl(50, 0.0, 1e-11, 1e6)
            s["P32"] = P32
        else:
            solver = b200.GMRES(pf, 30)
            solver.SetupOperator(P.A_perm)
            solver.SetupPreconditioner(P)
            solver.InitControl(10000, 0.0, 1e-10, 1e6)
        s.update(P=P, solver=solver, b=pf.vector(_rhs(2, N, seed)[P.perm]), x=pf.vector(len(row) - 1),
                 back=np.argsort(P.perm).astype(np.int32))
        return s
    dim, N = case["dim"], case["N"]
    row, col, val = b200.q1_assemble(dim, N, 0, _field(N, dim, _sigma(case), 0.1, seed))
    n, bh = len(row) - 1, _rhs(dim, N, seed)
    if kind == "mcsgs":
        P = b200.Preconditioner.MultiColoringSGS(pf, row, col, val)
        A, bh = P.A_perm, bh[P.perm]
    else:
        A = b200.CSR_lMatrix.from_csr(pf, row, col, val)
        P = b200.Preconditioner.Jacobi(pf, A) if kind == "pcg" else None
    s.update(A=A, P=P, b=pf.vector(bh), x=pf.vector(n))
    if kind in ("pcg", "mcsgs"):
        s["solver"] = b200.CG(pf)
        s["solver"].SetupOperator(A)
        s["solver"].SetupPreconditioner(P)
        s["solver"].InitControl(100000, 0.0, 1e-12, 1e6)
    elif kind == "mpir":
        s["solver"] = b200.MPIR(pf)
        s["solver"].SetupOperator(A)
        s["A32"] = A.CastFrom(b200.F32)
        s["solver"].SetupLowPrecisionOperator(s["A32"])
        s["solver"].InitControl(50, 0.0, 1e-11, 1e6)
    elif kind == "lmp_cg":
        s.update(r=pf.vector(n), p=pf.vector(n), Ap=pf.vector(n))
    else:
        r, c, v = _interp(dim, N // 2)
        nc = (N // 2 + 1) ** dim
        s.update(Pr=b200.CSR_lMatrix.from_csr(pf, *_to_csr(r, c, v, n), n_cols=nc),
                 R=b200.CSR_lMatrix.from_csr(pf, *_to_csr(c, r, v * 0.5 ** dim, nc), n_cols=n),
                 sol=pf.vector(np.random.default_rng(seed + 9).uniform(-1, 1, n)),
                 e=pf.vector(np.random.default_rng(seed + 11).uniform(-1, 1, nc)), r=pf.vector(n), rc=pf.vector(nc))
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "serve":
        return s["served"].run()
    if kind == "spmv":
        s["A"].VectorMult(s["x"], s["y"])
        return s["y"].t
    if kind == "lmp_cg":
        return _host_cg(s)
    if kind == "gmg":
        b200, x = _package(), s["x"]
        x.CopyFrom(s["sol"])
        b200.gmg_residual(s["pf"], s["A"], x, s["b"], s["r"])
        b200.gmg_restriction(s["pf"], s["R"], s["r"], s["rc"])
        b200.gmg_prolongation_add(s["pf"], s["Pr"], s["e"], x)
        return {"r": s["r"].t, "rc": s["rc"].t, "x": x.t}
    s["x"].Zeros()
    s["solver"].Solve(s["b"], s["x"])
    if kind == "gmres":      # the solution read back in the grid's numbering
        return s["x"].GetIndexedValues(s["back"])
    return s["x"].t


def _host_cg(s):
    """Unpreconditioned CG as a host program writes it over lMatrix / lVector."""
    A, b, x, r, p, Ap = (s[k] for k in ("A", "b", "x", "r", "p", "Ap"))
    x.Zeros()
    r.CopyFrom(b)
    p.CopyFrom(r)
    rho = r.Dot(r)
    for _ in range(s["case"]["its"]):
        A.VectorMult(p, Ap)
        alpha = rho / p.Dot(Ap)
        x.Axpy(p, alpha)
        r.Axpy(Ap, -alpha)
        new = r.Dot(r)
        p.ScaleAdd(new / rho, r)
        rho = new
    return {"x": x.t, "r": r.t, "norm": r.Norm2()}


# ------------------------------------------------------------------ work

def work(case):
    """One pass's bytes and operations.  A solve streams its operator and its
    vectors once per iteration (symmetric grid operators: the diagonal and the
    upper half, no indices); the iteration counts are those of the sizes and
    tolerances above, to a few per cent."""
    kind = case["kind"]
    if kind == "serve":
        total = dict(bytes=0.0, flops=0.0)
        for q in _requests(case, 1):
            w = _cg_work(q["dim"], q["N"], q["mixed"], 11)
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "spmv":
        es = 4 if case["f32"] else 8
        nnz = case["n"] * case["mean"]
        return dict(bytes=nnz * (es + 4) + case["n"] * (4 + 2 * es), flops=2 * nnz)
    if kind == "gmres":
        n = (case["N"] + 1) ** 2
        es = 4 if case["mixed"] else 8
        its = (0.3 if case["p"] == 0 else 0.2) * case["N"] * (1.6 if case["mixed"] else 1.0) + 10
        fact = 9 if case["p"] == 0 else 13
        # product, factors, and on average half a basis of 30 read once per step
        return dict(bytes=its * n * es * (9 + fact + 6 + 15), flops=its * n * (18 + 2 * fact + 60))
    dim, N = case["dim"], case["N"]
    n, k = (N + 1) ** dim, 3 ** dim
    if kind == "lmp_cg":
        return dict(bytes=case["its"] * n * 8.0 * ((k + 1) // 2 + 13), flops=case["its"] * n * (2 * k + 10.0))
    if kind == "gmg":
        nc = (N // 2 + 1) ** dim
        stencil = (1.5 ** dim) * n
        return dict(bytes=8.0 * n * ((k + 1) // 2 + 4) + 2 * 12 * stencil + 8 * (3 * n + 2 * nc),
                    flops=2.0 * n * k + 4 * stencil)
    if kind == "mcsgs":
        its = (1.5 if dim == 3 else 1.8) * N
        return dict(bytes=its * n * 8.0 * (k - 1 + (k + 1) // 2 + 16), flops=its * n * (4 * k + 20.0))
    return _cg_work(dim, N, kind == "mpir", 12 if kind == "pcg" else 11)


def _cg_work(dim, N, mixed, digits):
    n, k = (N + 1) ** dim, 3 ** dim
    its = (2.4 if dim == 2 else 2.9) * N * digits / 10 * (1.2 if mixed else 1.0)
    return dict(bytes=its * n * (4.0 if mixed else 8.0) * ((k + 1) // 2 + 10), flops=its * n * (2 * k + 12.0))


# ------------------------------------------------------------------ exact values

def _q1_diagonals(dim, N, kcell=None, nu=1.0, beta=None):
    """{offset (dx[, dy, dz]): array over nodes} of the Q1 operator, Dirichlet
    rows set to identity rows, from the closed-form 1-D element matrices."""
    h = 1.0 / N
    M1 = np.array([[2.0, 1.0], [1.0, 2.0]]) * h / 6
    K1 = np.array([[1.0, -1.0], [-1.0, 1.0]]) / h
    C1 = np.array([[-0.5, 0.5], [-0.5, 0.5]])

    def kron(ms):          # element matrix, vertex index = sum of bit_d << d
        out = np.ones((1, 1))
        for m in reversed(ms):
            out = np.kron(out, m)
        return out

    Ke = sum(kron([K1 if e == d else M1 for e in range(dim)]) for d in range(dim))
    Ce = sum(beta[d] * kron([C1 if e == d else M1 for e in range(dim)]) for d in range(dim)) if beta else 0 * Ke
    kc = torch.full((N,) * dim, nu, dtype=torch.float64, device=DEV) if kcell is None else \
        torch.from_numpy(kcell).to(DEV).reshape((N,) * dim)
    inner = torch.from_numpy(_interior(dim, N)).to(DEV).reshape((N + 1,) * dim)
    D = {}
    for a in range(1 << dim):
        for b in range(1 << dim):
            o = tuple(((b >> d) & 1) - ((a >> d) & 1) for d in range(dim))
            if o not in D:
                D[o] = torch.zeros((N + 1,) * dim, dtype=torch.float64, device=DEV)
            at = tuple(slice((a >> d) & 1, ((a >> d) & 1) + N) for d in reversed(range(dim)))
            D[o][at] += Ke[a, b] * kc + Ce[a, b] if beta else Ke[a, b] * kc
    for o in D:
        D[o] = torch.where(inner, D[o], torch.full_like(D[o], 1.0 if not any(o) else 0.0))
    return D


def _apply(D, x, dim, N):
    xp = torch.nn.functional.pad(x, (1, 1) * dim)
    y = torch.zeros_like(x)
    for o, d in D.items():
        y.addcmul_(d, xp[tuple(slice(1 + o[k], 2 + o[k] + N) for k in reversed(range(dim)))])
    return y


def _solve_spd(dim, N, kcell, b):
    """CG in 64 bits until the residual no longer falls, then one correction."""
    D = _q1_diagonals(dim, N, kcell)
    bt = torch.from_numpy(b).to(DEV).reshape((N + 1,) * dim)
    dinv = 1.0 / D[(0,) * dim]
    x = torch.zeros_like(bt)
    for target in (1e-13, 1e-5):
        r = bt - _apply(D, x, dim, N)
        z = r * dinv
        p, rho, dx, stop = z.clone(), (r * z).sum(), torch.zeros_like(x), float(r.norm()) * target
        for it in range(20 * N):
            Ap = _apply(D, p, dim, N)
            alpha = rho / (p * Ap).sum()
            dx += alpha * p
            r -= alpha * Ap
            z = r * dinv
            new = (r * z).sum()
            p = z + (new / rho) * p
            rho = new
            if it % 20 == 19 and float(r.norm()) <= stop:
                break
        x = x + dx
    return x.reshape(-1)


def _solve_lines(D, N, b):
    """Block elimination by grid lines (the nonsymmetric 2-D operator), refined twice."""
    def line(dy, j):
        m = torch.diag(D[(0, dy)][j])
        m += torch.diag(D[(1, dy)][j, :-1], 1) + torch.diag(D[(-1, dy)][j, 1:], -1)
        return m

    bt = torch.from_numpy(b).to(DEV).reshape(N + 1, N + 1)
    lu, W = [], []
    for j in range(N + 1):
        S = line(0, j) if j == 0 else line(0, j) - line(-1, j) @ W[-1]
        lu.append(torch.linalg.lu_factor(S))
        W.append(torch.linalg.lu_solve(*lu[-1], line(1, j)) if j < N else None)
    x = torch.zeros_like(bt)
    for _ in range(3):
        r = bt - _apply(D, x, 2, N)
        g = []
        for j in range(N + 1):
            t = r[j] if j == 0 else r[j] - line(-1, j) @ g[-1]
            g.append(torch.linalg.lu_solve(*lu[j], t[:, None])[:, 0])
        for j in range(N - 1, -1, -1):
            g[j] = g[j] - W[j] @ g[j + 1]
        x = x + torch.stack(g)
    return x.reshape(-1)


def _coords(dim, N):
    g = np.meshgrid(*[np.arange(N + 1)] * dim, indexing="ij")
    return [a.reshape(-1) for a in reversed(g)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        # every sixth solution: two- and three-dimensional systems in turn come up
        return [_solve_spd(q["dim"], q["N"], _field(q["N"], 2, 0.5, 0.1, q["seed"]) if q["dim"] == 2 else None,
                           _rhs(q["dim"], q["N"], q["seed"])) if k % 6 == 4 else None
                for k, q in enumerate(_requests(case, seed))]
    if kind == "spmv":
        row, col, val, x = _csr_unstructured(case, seed)
        if case["f32"]:
            val, x = val.astype(np.float32).astype(np.float64), x.astype(np.float32).astype(np.float64)
        return np.add.reduceat(val * x[col], row[:-1].astype(np.int64))
    if kind == "gmres":
        N = case["N"]
        return _solve_lines(_q1_diagonals(2, N, None, GMRES_NU, GMRES_BETA), N, _rhs(2, N, seed))
    dim, N = case["dim"], case["N"]
    kc, b = _field(N, dim, _sigma(case), 0.1, seed), _rhs(case["dim"], N, seed)
    if kind == "lmp_cg":
        D = _q1_diagonals(dim, N, kc)
        r = torch.from_numpy(b).to(DEV).reshape((N + 1,) * dim)
        x, p, rho = torch.zeros_like(r), r.clone(), (r * r).sum()
        for _ in range(case["its"]):
            Ap = _apply(D, p, dim, N)
            alpha = rho / (p * Ap).sum()
            x = x + alpha * p
            r = r - alpha * Ap
            new = (r * r).sum()
            p = r + (new / rho) * p
            rho = new
        return {"x": x.reshape(-1), "r": r.reshape(-1), "norm": float(rho.sqrt())}
    if kind == "gmg":
        n, nc = (N + 1) ** dim, (N // 2 + 1) ** dim
        x = torch.from_numpy(np.random.default_rng(seed + 9).uniform(-1, 1, n)).to(DEV)
        e = torch.from_numpy(np.random.default_rng(seed + 11).uniform(-1, 1, nc)).to(DEV)
        r, c, v = (torch.from_numpy(a).to(DEV) for a in _interp(dim, N // 2))
        D = _q1_diagonals(dim, N, kc)
        res = torch.from_numpy(b).to(DEV) - _apply(D, x.reshape((N + 1,) * dim), dim, N).reshape(-1)
        rc = torch.zeros(nc, dtype=torch.float64, device=DEV).index_add_(0, c, v * 0.5 ** dim * res[r])
        return {"r": res, "rc": rc, "x": x.index_add(0, r, v * e[c])}
    x = _solve_spd(dim, N, kc, b)
    if kind == "mcsgs":      # the colour numbering: node parities, lexicographic inside
        colour = sum((a % 2) << d for d, a in enumerate(_coords(dim, N)))
        x = x[torch.from_numpy(np.argsort(colour, kind="stable")).to(DEV)]
    return x
