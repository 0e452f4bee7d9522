"""Matrices of two scales (test_gpu_two_scales.py) through Arnoldi in one launch:
the window of the dots is not the one that ||A|| suggests, or changes by many
powers of two from step to step."""
import numpy as np
import pytest
import scipy.sparse as sp
from test_gpu_two_scales import both_scales, check, two_scales

from psfun_gb300 import matrices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [1e3, 1e6, 1e9, 1e12, 1e16, 1e20, 1e25, 1e60])
@pytest.mark.parametrize("at", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("istop", [1, 2])
def test_a_row_not_met(lib, orc, D, at, istop):
    check(orc, *two_scales(D, at), "ARNOLDI", "GENPADE", istop)


@pytest.mark.parametrize("scale", [1e-30, 1e-12])
def test_both_scales_met(lib, orc, scale):
    check(orc, *both_scales(scale), "ARNOLDI", "GENPADE", 2)


def test_above_the_bound(lib, orc):
    """A full column: ||A||_2 is 70 times ||A||_inf."""
    n = 5000
    A = sp.lil_matrix(1e-3 * matrices.laplacian_1d(n))
    A[:, 0] = 0.99
    x = np.zeros(n)
    x[0] = 1.0
    check(orc, sp.csr_matrix(A), x, "ARNOLDI", "GENPADE", 2, m=8)


@pytest.mark.parametrize("step", [-60, -30, -13, 13, 30])
def test_scale_changes_at_every_step(lib, orc, step):
    """A chain: step k reaches row k alone, whose entry is 2^step times the one
    before it (growing ones are capped at 2^60)."""
    n, m = 3000, 9
    e = np.minimum(2.0 ** (step * np.arange(n - 1.0).clip(max=20)), 2.0 ** 60) if step > 0 else \
        2.0 ** (step * np.arange(n - 1.0).clip(max=12))
    A = sp.csr_matrix(sp.diags([e * 1e-3], [-1], shape=(n, n)))
    x = np.zeros(n)
    x[0] = 1.0
    check(orc, A, x, "ARNOLDI", "GENPADE", 2, m=m)


@pytest.mark.parametrize("xs,As", [(1.0, 1e-156), (1e120, 1e-156)])
def test_scales_whose_product_overflows(lib, orc, xs, As):
    """1 / (||W_j|| ||W_k||) is beyond the largest double."""
    A = As * matrices.laplacian_2d(40)
    check(orc, sp.csr_matrix(A), xs * np.random.default_rng(2).standard_normal(1600), "ARNOLDI", "GENPADE", 2, m=12)


@pytest.mark.parametrize("delta", [1e-3, 1e-4, 1e-5, 1e-6, 1e-7])
def test_orthogonality_lost_by_degrees(lib, delta):
    """x is an eigenvector up to delta: the second basis vector has lost
    eps / delta of its orthogonality, on either side of where the coefficients'
    correction leaves FP32.  The result is exp(A) x all the same."""
    d = -np.linspace(0.0, 4.0, 4001)
    x = delta * np.random.default_rng(3).standard_normal(d.size)
    x[-1] = 1.0
    import psfun_gb300 as pg
    fun = pg.PsfunDSerial()
    assert fun.set("VARIANT", "GENPADE") == 0
    r = pg.PsfunDKrylov().apply(fun, pg.CsrMatrix.from_scipy(sp.diags(d).tocsr()), x, 1e-12, itmax=30, istop=2)
    y = np.exp(d) * x
    assert r.info == 0 and np.linalg.norm(r.y - y) <= 1e-10 * np.linalg.norm(y)
