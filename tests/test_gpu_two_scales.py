"""Matrices of two scales: a row of size D next to an operator of norm ~8, and
vectors that are zero in that row.  ||A|| = D then says nothing about the sums
of a step, which are those of the operator alone, and so is the result: D does
not enter it (D times zero is zero).  D = 0 is the same solve by the same code
with tight bounds; the oracle takes the matrix with D."""
import numpy as np
import pytest
import scipy.sparse as sp

from psfun_gb300 import matrices

pytestmark = pytest.mark.gpu
TOL = 1e-10


def two_scales(D, at, n1=60):
    """-(Laplacian) with one more row and column, -D on its diagonal, at the
    place `at` of the n1^2 + 1; the vector is zero there."""
    L = -matrices.laplacian_2d(n1)
    n = L.shape[0]
    k = int(at * n)
    A = sp.block_diag([L[:k, :k], sp.csr_matrix([[-D]]), L[k:, k:]], format="lil")
    A[:k, k + 1:] = L[:k, k:]
    A[k + 1:, :k] = L[k:, :k]
    x = np.random.default_rng(7).standard_normal(n + 1)
    x[k] = 0.0
    return sp.csr_matrix(A), x


def both_scales(scale):
    """Two uncoupled operators, both met by x: the sums are those of the large
    one and the small one must come out of the same basis."""
    L = -matrices.laplacian_2d(30)
    A = sp.csr_matrix(sp.block_diag([L, scale * L]))
    return A, np.random.default_rng(8).standard_normal(A.shape[0])


def check(orc, A, x, kname, variant, istop, m=30):
    import psfun_gb300 as pg
    fun, meth = pg.PsfunDSerial(), pg.PsfunDKrylov()
    assert fun.set("VARIANT", variant) == 0 and meth.set("KNAME", kname) == 0
    r = meth.apply(fun, pg.CsrMatrix.from_scipy(A), x, 1e-10, itmax=m, istop=istop)
    o = orc.krylov(kname, orc.serial("EXP", variant, 1.0), orc.Csr.from_scipy(A), x, 1e-10, itmax=m, istop=istop)
    assert r.info == 0 and o["info"] == 0 and r.iter == o["iter"]
    assert np.linalg.norm(r.y - o["y"]) <= TOL * np.linalg.norm(o["y"])


@pytest.mark.parametrize("D", [1e3, 1e6, 1e9, 1e12, 1e16, 1e20, 1e25, 1e60])
@pytest.mark.parametrize("at", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("istop", [1, 2])
def test_lanczos(lib, orc, D, at, istop):
    check(orc, *two_scales(D, at), "LANCZOS", "CHBSYM", istop)


@pytest.mark.parametrize("scale", [1e-30, 1e-12])
def test_lanczos_both_scales_met(lib, orc, scale):
    check(orc, *both_scales(scale), "LANCZOS", "CHBSYM", 2)


@pytest.mark.parametrize("n1", [25, 120])
def test_lanczos_alpha_zero(lib, orc, n1):
    """The adjacency of a grid (bipartite) from one vertex: every alpha is
    exactly zero, and most rows are zero at first."""
    L = matrices.laplacian_2d(n1)
    x = np.zeros(L.shape[0])
    x[L.shape[0] // 3] = 1.0
    check(orc, sp.csr_matrix(sp.diags(L.diagonal()) - L), x, "LANCZOS", "CHBSYM", 1)


def test_lanczos_above_the_bound(lib, orc):
    """A matrix that is not symmetric, with a full column: ||A|| is ~70 times
    ||A||_inf, and a block's part of the norm is above its bound."""
    n = 5000
    A = sp.lil_matrix(1e-3 * matrices.laplacian_1d(n))
    A[:, 0] = 0.99
    x = np.zeros(n)
    x[0] = 1.0
    check(orc, sp.csr_matrix(A), x, "LANCZOS", "GENPADE", 2, m=4)


@pytest.mark.parametrize("D", [1e12, 1e16, 1e25])
def test_quadrature(lib, D):
    torch = pytest.importorskip("torch")
    import psfun_gb300 as pg
    A, x = two_scales(D, 0.4, 30)
    lo, hi = 8.0 * np.sin(np.pi / 62.0) ** 2, 8.0
    q = pg.PsfunZQuadrature()
    assert q.computepoles(pg.hhtmethod1, lambda z: 1.0 / np.sqrt(z), 24, rparams=[0.9 * lo, 1.1 * hi]) == 0
    out = []
    for B in (-A, -two_scales(0.0, 0.4, 30)[0]):
        h = pg.CsrMatrix.from_scipy(sp.csr_matrix(B))
        q.setmatrix(h)
        y = torch.empty(x.size, dtype=torch.float64, device="cuda")
        y, info, it, _ = q.apply(torch.tensor(x, device="cuda"), eps=1e-12, itmax=300, y=y)
        assert info == 0
        out.append((y.cpu().numpy(), it))
    # the same solve up to rounding in T, whose relative effect the residuals (1e-12) bound
    assert out[0][1] == out[1][1]
    assert np.linalg.norm(out[0][0] - out[1][0]) <= TOL * np.linalg.norm(out[1][0])


@pytest.mark.parametrize("D", [1e12, 1e16, 1e25])
def test_adjoint(lib, D):
    torch = pytest.importorskip("torch")
    import psfun_gb300 as pg
    out = []
    A0, x = two_scales(0.0, 0.4, 30)
    g = np.roll(x, 17)
    g[x == 0.0] = 0.0
    for d in (D, 0.0):
        A = two_scales(d, 0.4, 30)[0]
        # d = 0 keeps the pattern: the entry is stored explicitly
        if d == 0.0:
            B = two_scales(1.0, 0.4, 30)[0]
            B.data[B.data == -1.0] = 0.0
            A = B
        r = pg.expm_adjoint(pg.CsrMatrix.from_scipy(A), 0.1, torch.tensor(x, device="cuda"),
                            torch.tensor(g, device="cuda"))
        out.append([r["y"].cpu().numpy(), r["grad_x"].cpu().numpy(), r["grad_vals"].cpu().numpy(),
                    np.array([r["grad_t"]])])
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)
