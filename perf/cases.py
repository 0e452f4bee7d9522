"""The work a user of psfun_gb300 has it do, as timed cases.

Nine kinds, each through its public entry point:

  lanczos     PsfunDKrylov.apply, KNAME LANCZOS   y = exp(-tA) x, A symmetric
  arnoldi     PsfunDKrylov.apply, KNAME ARNOLDI   y = f(-tA) x, exp or phi_1
  quadrature  PsfunZQuadrature.apply              y = A^{-1/2} x by a conformal-map rule
  cg          psb_krylov                          (A + zeta I) x = b
  adjoint     expm_adjoint                        exp(tA) x and every gradient
  batch       krylov_batch                        uneven instances, several right-hand sides each
  serial      PsfunDSerial.apply                  dense f(H) x of a small H, host arrays
  spmv        CsrMatrix.spmv                      y = A x

Matrices are the ones of this repository's drivers, tests and benchmark: 2-D and
3-D grid Laplacians (constant or lognormal conductivities), the 2-D upwind
convection-diffusion operator, k-nearest-neighbour graph Laplacians and
power-law row lengths.  Grids have their own side per axis, so that odd and
uneven ones occur.  Inputs come from the seed; a case's sizes do not.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import psfun_gb300 as pg
from psfun_gb300 import matrices

DEV = "cuda"


def listed():
    return [
        # The reference's own example size: a 100 x 100 Laplacian to a
        # tolerance.  A call of a fraction of a millisecond, all latency.
        dict(name="lanczos_grid_100", kind="lanczos", nx=100, ny=100, nz=1, coef="unit", t=1.0, m=50, eps=1e-10,
             istop=1),
        # A production-size diffusion step: a fixed Krylov space on a 3-D grid
        # whose matrix and basis are far larger than L2.
        dict(name="lanczos_cube_128", kind="lanczos", nx=128, ny=128, nz=128, coef="unit", t=0.05, m=80, eps=1e-12,
             istop=2),
        # The same example through Arnoldi and the dense Pade exponential.
        dict(name="arnoldi_grid_100", kind="arnoldi", nx=100, ny=100, fname="EXP", beta=0.0, t=1.0, m=50, eps=1e-10,
             istop=1),
        # An exponential-integrator stage, phi_1, on a nonsymmetric operator of
        # ordinary and odd size.
        dict(name="arnoldi_phi_301", kind="arnoldi", nx=301, ny=287, fname="PHI", beta=50.0, t=1e-4, m=40, eps=1e-12,
             istop=2),
        # The same stage at the largest size: a basis of two gigabytes.
        dict(name="arnoldi_phi_2048", kind="arnoldi", nx=2048, ny=2048, fname="PHI", beta=50.0, t=1e-3, m=60,
             eps=1e-12, istop=2),
        # Sampling with a precision matrix: A^{-1/2} x, hundreds of short
        # Lanczos steps and 24 shifted systems.
        dict(name="quad_cube_96", kind="quadrature", nx=96, ny=96, nz=96, N=24, eps=1e-10),
        # One implicit time step: shifted CG with the cheap preconditioner.
        dict(name="cg_diag_cube_128", kind="cg", nx=128, ny=128, nz=128, coef="unit", prec="DIAG", zeta=0.5, eps=1e-10),
        # The same with the strong preconditioner, on an uneven grid with
        # jumping coefficients, where one is wanted.
        dict(name="cg_bjac_grid_701", kind="cg", nx=701, ny=613, nz=1, coef="lognormal", prec="BJAC", zeta=0.05,
             eps=1e-10),
        # Forward and backward of a diffusion layer: gradients with respect to
        # x, t and every conductivity.
        dict(name="adjoint_grid_512", kind="adjoint", nx=512, ny=512, t=0.1),
        # Many graphs at once: grids and neighbour graphs of very different
        # sizes, four signals each.
        dict(name="batch_graphs_24", kind="batch", count=24, nrhs=4, nmin=4096, nmax=65536, m=60, eps=1e-8),
        # The dense function alone, called on host arrays by the drivers.
        dict(name="serial_pade_80", kind="serial", n=80, variant="GENPADE"),
        # The product alone, on rows of power-law length.
        dict(name="spmv_skewed_1m", kind="spmv", n=1000003, alpha=1.5),
    ]


# The kinds as often as they are listed.
_KINDS = ("lanczos", "lanczos", "arnoldi", "arnoldi", "arnoldi", "quadrature", "cg", "cg", "adjoint", "batch", "serial",
          "spmv")


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, nlo, nhi, dim):
    """Uneven sides whose product is log-uniform over [nlo, nhi]."""
    n = math.exp(rng.uniform(math.log(nlo), math.log(nhi)))
    s = n ** (1.0 / dim)
    f = [rng.uniform(0.8, 1.0) for _ in range(dim)]
    return [max(3, int(s * v)) for v in f] + [1] * (3 - dim)


def draw(rng):
    kind = rng.choice(_KINDS)
    if kind == "lanczos":
        nx, ny, nz = _sides(rng, 5000, 2.1e6, rng.choice((2, 3)))
        coef = rng.choice(("unit", "lognormal"))
        c = dict(kind=kind, nx=nx, ny=ny, nz=nz, coef=coef, t=round(math.exp(rng.uniform(math.log(0.05), 0.0)), 4))
        if rng.random() < 0.5:
            return dict(c, m=200, eps=rng.choice((1e-6, 1e-8, 1e-10)), istop=1)
        return dict(c, m=rng.randint(20, 80), eps=1e-12, istop=2)
    if kind == "arnoldi":
        if rng.random() < 0.35:  # to a tolerance, small
            nx, ny, _ = _sides(rng, 1000, 60000, 2)
            return dict(kind=kind, nx=nx, ny=ny, fname="EXP", beta=0.0, t=round(rng.uniform(0.2, 1.5), 3), m=60,
                        eps=rng.choice((1e-8, 1e-10)), istop=1)
        nx, ny, _ = _sides(rng, 10000, 4.2e6, 2)
        norm = 8.0 * max(nx, ny) ** 2
        return dict(kind=kind, nx=nx, ny=ny, fname="PHI", beta=round(rng.uniform(5.0, 100.0), 1),
                    t=float("%.3g" % (math.exp(rng.uniform(math.log(4.0), math.log(3e4))) / norm)),
                    m=rng.randint(10, 60), eps=1e-12, istop=2)
    if kind == "quadrature":
        nx, ny, nz = _sides(rng, 8000, 884736, 3)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, N=rng.choice((8, 12, 16, 24)), eps=rng.choice((1e-8, 1e-10)))
    if kind == "cg":
        nx, ny, nz = _sides(rng, 10000, 2.1e6, rng.choice((2, 3)))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, coef=rng.choice(("unit", "lognormal")),
                    prec=rng.choice(("NONE", "DIAG", "BJAC")), zeta=round(rng.uniform(0.05, 1.0), 3), eps=1e-10)
    if kind == "adjoint":
        nx, ny, _ = _sides(rng, 4096, 262144, 2)
        return dict(kind=kind, nx=nx, ny=ny, t=round(rng.uniform(0.05, 0.2), 3))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 24), nrhs=rng.choice((1, 2, 4)), nmin=2048,
                    nmax=_logint(rng, 8192, 65536), m=60, eps=1e-8)
    if kind == "serial":
        return dict(kind=kind, n=_logint(rng, 5, 100),
                    variant=rng.choice(("GENPADE", "GENPADE", "CHBGEN", "CHBSYM", "TAYLOR")))
    return dict(kind="spmv", n=_logint(rng, 20000, 1000000), alpha=round(rng.uniform(1.4, 2.5), 2))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1000003 + salt)


def _normal(n, seed, salt=0):
    return torch.randn(n, generator=_gen(seed, salt), dtype=torch.float64, device=DEV)


def _unit(v):
    return v / torch.linalg.norm(v)


def _stencil(dims, diag, lo, up):
    """CSR of a grid stencil, x fastest: diag and, per axis, the coefficients
    of the lower and the upper neighbour (numbers or one value per row)."""
    n = math.prod(dims)
    idx = torch.arange(n, device=DEV)
    stride = [math.prod(dims[:k]) for k in range(len(dims))]
    cols, vals, here = [], [], []
    for k in reversed(range(len(dims))):
        if dims[k] > 1:
            cols.append(idx - stride[k])
            vals.append(lo[k])
            here.append((idx // stride[k]) % dims[k] > 0)
    cols.append(idx)
    vals.append(diag)
    here.append(torch.ones_like(idx, dtype=torch.bool))
    for k in range(len(dims)):
        if dims[k] > 1:
            cols.append(idx + stride[k])
            vals.append(up[k])
            here.append((idx // stride[k]) % dims[k] < dims[k] - 1)
    full = [v if torch.is_tensor(v) else torch.full((n,), float(v), dtype=torch.float64, device=DEV) for v in vals]
    mask = torch.stack(here, 1)
    irp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    irp[1:] = torch.cumsum(mask.sum(1), 0)
    return irp.int(), torch.stack(cols, 1)[mask].int(), torch.stack(full, 1)[mask].contiguous()


def _laplacian(dims, coef, seed, scale=1.0):
    """scale * the Dirichlet grid Laplacian (unit), or the Laplacian of the grid
    graph with lognormal(0, 0.7) conductivities (lognormal)."""
    d = sum(1 for s in dims if s > 1)
    if coef == "unit":
        return _stencil(dims, 2.0 * d * scale, [-scale] * 3, [-scale] * 3)
    n = math.prod(dims)
    idx = torch.arange(n, device=DEV)
    diag = torch.zeros(n, dtype=torch.float64, device=DEV)
    lo, up = [0.0] * 3, [0.0] * 3
    for k in range(len(dims)):
        if dims[k] == 1:
            continue
        st = math.prod(dims[:k])
        w = torch.exp(0.7 * _normal(n, seed, 17 + k))  # the edge to the upper neighbour
        w = torch.where((idx // st) % dims[k] < dims[k] - 1, w, 0.0)
        below = torch.zeros_like(w)
        below[st:] = w[:-st]
        below = torch.where((idx // st) % dims[k] > 0, below, 0.0)
        up[k], lo[k] = -scale * w, -scale * below
        diag += scale * (w + below)
    return _stencil(dims, diag, lo, up)


def _convdiff(nx, ny, beta, scale=1.0):
    """scale * (-Lap u + (beta, beta/2) . grad u), first-order upwind, on the
    unit square; beta = 0: the unscaled 5-point Laplacian."""
    if beta == 0.0:
        return _laplacian([nx, ny], "unit", 0, scale)
    hx, hy, bx, by = 1.0 / (nx + 1), 1.0 / (ny + 1), beta, beta / 2
    lo = [-scale * (1 / hx**2 + bx / hx), -scale * (1 / hy**2 + by / hy)]
    up = [-scale / hx**2, -scale / hy**2]
    return _stencil([nx, ny], -sum(lo) - sum(up), lo, up)


def _handle(csr):
    irp, ja, val = csr
    return pg.CsrMatrix(irp.cpu().numpy(), ja.cpu().numpy(), val.cpu().numpy())


def _batch_sizes(case):
    """Half grids, half neighbour graphs, rows log-uniform over [nmin, nmax];
    set by the case alone."""
    rng = random.Random(case["count"] * 7 + case["nmax"])
    out = []
    for k in range(case["count"]):
        n = _logint(rng, case["nmin"], case["nmax"])
        t = rng.uniform(0.01, 1.0)
        out.append(("graph", n, 1, t) if k % 2 else ("grid", int(math.sqrt(n)), int(math.sqrt(n)) + k % 5, t))
    return out


def _batch_matrix(kind, p, q, seed, k):
    """Host CSR arrays of one instance."""
    if kind == "grid":
        return tuple(v.cpu().numpy() for v in _laplacian([p, q], "unit", 0))
    A = matrices.rgg_knn_laplacian(p, 8, np.random.default_rng(seed * 131 + k))
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data


def _serial_inputs(case, seed):
    rng = np.random.default_rng(seed)
    B = rng.standard_normal((case["n"], case["n"]))
    H = -2.5 * (B @ B.T / case["n"] + np.eye(case["n"]))
    return H, rng.standard_normal(case["n"])


def _skewed(case, seed):
    """Rows of power-law length 4 .. 4000, random columns (sorted, distinct)."""
    n = case["n"]
    u = 1.0 - torch.rand(n, generator=_gen(seed, 3), dtype=torch.float64, device=DEV)
    lens = torch.clamp((4.0 * u ** (-1.0 / case["alpha"])).long(), max=min(4000, n))
    row = torch.repeat_interleave(torch.arange(n, device=DEV), lens)
    col = torch.randint(0, n, row.shape, generator=_gen(seed, 4), device=DEV)
    key = torch.unique(row * n + col)
    row, col = key // n, key % n
    irp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    irp[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    return irp.int(), col.int(), _normal(col.shape[0], seed, 5)


def _dims(case):
    return [case["nx"], case["ny"], case.get("nz", 1)]


def _bounds(dims):
    """Extreme eigenvalues of the unit Dirichlet grid Laplacian."""
    lam = lambda k, s: 4.0 * math.sin(math.pi * k / (2.0 * (s + 1))) ** 2  # noqa: E731
    return sum(lam(1, s) for s in dims if s > 1), sum(lam(s, s) for s in dims if s > 1)


def _csr(case, seed):
    """The case's matrix as the entry point is given it."""
    kind = case["kind"]
    if kind == "lanczos":  # Lanczos takes -tA: it has no scaling of its own
        return _laplacian(_dims(case), case["coef"], seed, -case["t"])
    if kind == "arnoldi":
        return _convdiff(case["nx"], case["ny"], case["beta"])
    if kind == "quadrature":
        return _laplacian(_dims(case), "unit", seed)
    if kind == "cg":
        return _laplacian(_dims(case), case["coef"], seed)
    if kind == "adjoint":
        return _laplacian(_dims(case), "lognormal", seed)
    return _skewed(case, seed)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind == "serial":
        fun = pg.PsfunDSerial()
        fun.set("VARIANT", case["variant"])
        s["fun"], (s["H"], s["x"]) = fun, _serial_inputs(case, seed)
        return s
    if kind == "batch":
        fun, meth = pg.PsfunDSerial(), pg.PsfunDKrylov()
        fun.set("VARIANT", "CHBSYM")
        meth.set("KNAME", "LANCZOS")
        items = []
        for k, (g, p, q, t) in enumerate(_batch_sizes(case)):
            X = _normal((case["nrhs"], p * q), seed, k)
            items.append((pg.CsrMatrix(*_batch_matrix(g, p, q, seed, k)), X, torch.empty_like(X), -t))
        s.update(fun=fun, meth=meth, items=items)
        return s
    s["a"] = _handle(_csr(case, seed))
    n = s["a"].n
    if kind == "spmv":
        s["x"], s["y"] = _normal(n, seed), torch.empty(n, dtype=torch.float64, device=DEV)
        return s
    s["x"] = _normal(n, seed)
    s["y"] = torch.empty_like(s["x"])
    if kind in ("lanczos", "arnoldi"):
        s["x"] = _unit(s["x"])
        fun, meth = pg.PsfunDSerial(), pg.PsfunDKrylov()
        meth.set("KNAME", kind.upper())
        if kind == "lanczos":
            fun.set("VARIANT", "CHBSYM")
        else:
            fun.set("FNAME", case["fname"])
            fun.set("VARIANT", "GENPADE")
            fun.set("SCALING", -case["t"])
        s.update(fun=fun, meth=meth)
    elif kind == "quadrature":
        q = pg.PsfunZQuadrature()
        q.computepoles(pg.hhtmethod1, lambda z: 1.0 / np.sqrt(z), case["N"], rparams=list(_bounds(_dims(case))))
        q.setmatrix(s["a"])
        s["q"] = q
    elif kind == "adjoint":
        s["g"] = _normal(n, seed, 1)
    return s


def run(s):
    kind, c = s["kind"], s["case"]
    if kind in ("lanczos", "arnoldi"):
        r = s["meth"].apply(s["fun"], s["a"], s["x"], c["eps"], itmax=c["m"], istop=c["istop"], y=s["y"])
        return {"y": r.y, "iter": r.iter, "info": r.info}
    if kind == "quadrature":
        y, info, it, _ = s["q"].apply(s["x"], eps=c["eps"], itmax=2000, y=s["y"])
        return {"y": y, "info": info, "iter": it}
    if kind == "cg":
        s["y"].zero_()  # the initial guess
        x, info, it, _ = pg.psb_krylov("CG", s["a"], c["prec"], s["x"], 1.0, c["zeta"], s["y"], c["eps"], itmax=5000)
        return {"x": x, "info": info, "iter": it}
    if kind == "adjoint":
        o = pg.expm_adjoint(s["a"], -c["t"], s["x"], s["g"])
        return {"y": o["y"], "grad_x": o["grad_x"], "grad_t": o["grad_t"], "grad_vals": o["grad_vals"]}
    if kind == "batch":
        info, infos, iters, _ = pg.krylov_batch(s["meth"], s["fun"], s["items"], c["eps"], itmax=c["m"], istop=1)
        return {"Y": [it[2] for it in s["items"]], "info": info, "infos": infos, "iters": iters}
    if kind == "serial":
        y, info = s["fun"].apply(s["H"], s["x"])
        return {"y": y, "info": info}
    return s["a"].spmv(s["x"], y=s["y"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _grid_nnz(dims):
    n = math.prod(dims)
    return n + sum(2 * (n - n // s) for s in dims if s > 1)


def _exp_steps(rho, eps):
    """Lanczos steps for exp on an interval of half-length rho, from the
    a-priori bound 10 exp(-rho) (e rho / k)^k."""
    k = 2
    while k < 200 and math.log(10.0) - rho + k * (1.0 + math.log(max(rho, 1e-3) / k)) > math.log(eps):
        k += 1
    return k


def work(case):
    """Bytes: a Krylov step needs the whole result of the step before, so every
    step passes over the matrix (12 bytes an entry, 4 a row) and over the
    vectors it combines; the basis is read once more for the result.  Flops: two
    per stored entry and per vector element combined or dotted.  Steps to a
    tolerance are estimated."""
    kind = case["kind"]
    if kind == "serial":  # one exponential: about ten products and a solve
        n = case["n"]
        return {"bytes": 8.0 * (n * n + 2 * n), "flops": 22.0 * n**3}
    if kind == "spmv":
        nnz = case["n"] * 4.0 * case["alpha"] / (case["alpha"] - 1.0) * (0.96 if case["alpha"] < 1.8 else 1.0)
        return {"bytes": 12 * nnz + 20.0 * case["n"], "flops": 2 * nnz}
    if kind == "batch":
        b = f = 0.0
        for g, p, q, t in _batch_sizes(case):
            n, R = p * q, case["nrhs"]
            nnz = 11.0 * n if g == "graph" else _grid_nnz([p, q])
            k = _exp_steps(t * (11.0 if g == "graph" else 4.0), case["eps"])
            b += k * (12 * nnz + 4 * n + R * 40.0 * n) + R * 8.0 * n * (k + 1)
            f += R * (k * (2 * nnz + 8 * n) + 2.0 * n * k)
        return {"bytes": b, "flops": f}
    n, nnz = math.prod(_dims(case)), _grid_nnz(_dims(case))
    spmv = 12.0 * nnz + 4 * n + 16 * n
    if kind == "lanczos":
        L = 2 * sum(1 for s in _dims(case) if s > 1) * (1.0 if case["coef"] == "unit" else 4.0)
        k = case["m"] if case["istop"] == 2 else min(case["m"], _exp_steps(case["t"] * L, case["eps"]))
        return {"bytes": k * (spmv + 32 * n) + 8 * n * (k + 1), "flops": k * (2.0 * nnz + 8 * n) + 2.0 * n * k}
    if kind == "arnoldi":
        k = case["m"] if case["istop"] == 2 else min(case["m"], _exp_steps(4 * case["t"], case["eps"]))
        return {"bytes": sum(spmv + 8.0 * n * i + 16 * n for i in range(1, k)) + 8.0 * n * (k + 1),
                "flops": sum(2.0 * nnz + 4.0 * n * i + 2 * n for i in range(1, k)) + 2.0 * n * k}
    if kind == "quadrature":
        lo, hi = _bounds(_dims(case))
        k = 0.3 * math.sqrt(hi / lo) * math.log(2 / case["eps"])
        return {"bytes": k * (spmv + 32 * n) + 8 * n * (k + 1), "flops": k * (2.0 * nnz + 10 * n)}
    if kind == "cg":
        d = 4 * sum(1 for s in _dims(case) if s > 1) * (1.0 if case["coef"] == "unit" else 2.0)
        k = 0.5 * math.sqrt((d + case["zeta"]) / case["zeta"]) * math.log(2 / case["eps"])
        k *= 0.6 if case["prec"] == "BJAC" else 1.0
        return {"bytes": k * (spmv + 88 * n), "flops": k * (2.0 * nnz + 12 * n)}
    k = 18  # adjoint: two bases, their projected solves, the products on the pattern
    return {"bytes": 2 * k * (spmv + 32 * n) + 8.0 * (2 * n * (k + 1) + nnz + 3 * n),
            "flops": 2 * k * (2.0 * nnz + 10 * n) + 2.0 * n * k * k + 2.0 * nnz * k}


# ---------------------------------------------------------------------------
# The same results from plain torch in 64 bits
# ---------------------------------------------------------------------------
def _sparse(csr):
    irp, ja, val = csr
    n = irp.shape[0] - 1
    return torch.sparse_csr_tensor(irp.long(), ja.long(), val, (n, n))


def _rowsum_abs(csr):
    irp, _, val = csr
    c = torch.zeros(val.shape[0] + 1, dtype=torch.float64, device=DEV)
    c[1:] = torch.cumsum(val.abs(), 0)
    return float((c[irp[1:].long()] - c[irp[:-1].long()]).max())


def _expm_cheb(S, bound, t, X):
    """exp(-t A) X for symmetric A with spectrum in [0, bound], S = A: the
    Chebyshev series, its coefficients by the cosine rule."""
    M = 40 + int(4 * t * bound)
    th = (np.arange(M) + 0.5) * math.pi / M
    f = np.exp(-t * bound * 0.5 * (np.cos(th) + 1.0))
    c = [2.0 / M * float(np.dot(f, np.cos(j * th))) for j in range(M)]
    c[0] *= 0.5
    op = lambda V: (S @ V) * (2.0 / bound) - V  # noqa: E731
    T0, T1 = X, op(X)
    Y = c[0] * T0 + c[1] * T1
    for j in range(2, M):
        if abs(c[j]) < 1e-18 and j > t * bound:
            break
        T0, T1 = T1, 2.0 * op(T1) - T0
        Y = Y + c[j] * T1
    return Y


def _arnoldi_plain(S, scale, x, m, phi):
    """beta V f(H) e_1 on the Krylov space of dimension m - 2, the dimension the
    reference's fixed-length loop evaluates f on: classical Gram-Schmidt, twice."""
    k = m - 2
    V = torch.zeros((k + 1, x.shape[0]), dtype=torch.float64, device=DEV)
    H = torch.zeros((k + 1, k + 1), dtype=torch.float64)
    beta = float(torch.linalg.norm(x))
    V[0] = x / beta
    for j in range(k):
        w = scale * (S @ V[j])
        for _ in range(2):
            h = V[: j + 1] @ w
            w = w - h @ V[: j + 1]
            H[: j + 1, j] += h.cpu()
        H[j + 1, j] = float(torch.linalg.norm(w))
        V[j + 1] = w / H[j + 1, j].item()
    if phi:
        B = torch.zeros((k + 1, k + 1), dtype=torch.float64)
        B[:k, :k], B[0, k] = H[:k, :k], 1.0
        f = torch.linalg.matrix_exp(B)[:k, k]
    else:
        f = torch.linalg.matrix_exp(H[:k, :k])[:, 0]
    return beta * (f.to(DEV) @ V[:k])


def _sine(s):
    k = torch.arange(1, s + 1, dtype=torch.float64, device=DEV)
    Q = math.sqrt(2.0 / (s + 1)) * torch.sin(torch.outer(k, k) * (math.pi / (s + 1)))
    return 4.0 * torch.sin(math.pi * k / (2.0 * (s + 1))) ** 2, Q


def _laplacian_fun(dims, x, f):
    """f(L) x for the unit Dirichlet grid Laplacian through its sine basis."""
    nx, ny, nz = dims
    (lx, Qx), (ly, Qy), (lz, Qz) = _sine(nx), _sine(ny), _sine(nz)
    X = torch.einsum("ck,bj,ai,kji->cba", Qz, Qy, Qx, x.reshape(nz, ny, nx))
    X = X * f(lz[:, None, None] + ly[None, :, None] + lx[None, None, :])
    return torch.einsum("ck,bj,ai,kji->cba", Qz, Qy, Qx, X).reshape(-1)


def _cg_plain(S, dinv, zeta, b):
    x, r = torch.zeros_like(b), b.clone()
    z = dinv * r
    p, rz = z.clone(), torch.dot(r, z)
    for _ in range(4000):
        q = S @ p + zeta * p
        al = rz / torch.dot(p, q)
        x, r = x + al * p, r - al * q
        if float(torch.linalg.norm(r)) < 1e-14 * float(torch.linalg.norm(b)):
            break
        z = dinv * r
        rz, old = torch.dot(r, z), rz
        p = z + (rz / old) * p
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "serial":
        H, x = _serial_inputs(case, seed)
        return {"y": torch.linalg.matrix_exp(torch.from_numpy(H)) @ torch.from_numpy(x), "info": None}
    if kind == "batch":
        Y = []
        for k, (g, p, q, t) in enumerate(_batch_sizes(case)):
            csr = tuple(torch.as_tensor(v, device=DEV) for v in _batch_matrix(g, p, q, seed, k))
            X = _normal((case["nrhs"], p * q), seed, k)
            Y.append(_expm_cheb(_sparse(csr), _rowsum_abs(csr), t, X.T.contiguous()).T.contiguous())
        return {"Y": Y, "info": None, "infos": None, "iters": None}
    csr = _csr(case, seed)
    S, n = _sparse(csr), csr[0].shape[0] - 1
    x = _normal(n, seed)
    if kind == "spmv":
        return S @ x
    if kind == "lanczos":
        neg = (csr[0], csr[1], -csr[2])
        return {"y": _expm_cheb(_sparse(neg), _rowsum_abs(neg), 1.0, _unit(x)), "iter": None, "info": None}
    if kind == "arnoldi":
        if case["istop"] == 1:
            y = _expm_cheb(S, _rowsum_abs(csr), case["t"], _unit(x))
        else:
            y = _arnoldi_plain(S, -case["t"], _unit(x), case["m"], case["fname"] == "PHI")
        return {"y": y, "iter": None, "info": None}
    if kind == "quadrature":
        return {"y": _laplacian_fun(_dims(case), x, torch.rsqrt), "info": None, "iter": None}
    if kind == "cg":
        row = torch.repeat_interleave(torch.arange(n, device=DEV), (csr[0][1:] - csr[0][:-1]).long())
        d = csr[2][csr[1].long() == row] + case["zeta"]
        return {"x": _cg_plain(S, 1.0 / d, case["zeta"], x), "info": None, "iter": None}
    t, bound, g = case["t"], _rowsum_abs(csr), _normal(n, seed, 1)
    y, gx = _expm_cheb(S, bound, t, x), _expm_cheb(S, bound, t, g)
    # dL/dA = -t int_0^1 exp(-(1-s) tA) g (exp(-s tA) x)^T ds on the pattern
    row = torch.repeat_interleave(torch.arange(n, device=DEV), (csr[0][1:] - csr[0][:-1]).long())
    col, gv = csr[1].long(), torch.zeros_like(csr[2])
    node, wt = np.polynomial.legendre.leggauss(24)
    for u, w in zip(0.5 * (node + 1.0), 0.5 * wt):
        G, X = _expm_cheb(S, bound, (1.0 - u) * t, g), _expm_cheb(S, bound, u * t, x)
        gv -= t * w * G[row] * X[col]
    return {"y": y, "grad_x": gx, "grad_t": float(torch.dot(g, S @ y)), "grad_vals": gv}
