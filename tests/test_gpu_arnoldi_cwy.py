"""Arnoldi solves of fewer than 2^19 rows (k_ar_cwy: all coefficients of a step
from one set of grid sums) against the oracle's modified Gram-Schmidt, at the
edges of its row groups, of its two basis placements and of its fixed-point
windows.  Tolerance 1e-10 relative, as for every Krylov result here."""
import numpy as np
import pytest
import scipy.sparse as sp

from psfun_gb300 import matrices

pytestmark = pytest.mark.gpu
TOL = 1e-10


def solve(lib, A, x, m, scaling=-1.0, istop=2, eps=1e-10, variant="GENPADE"):
    import psfun_gb300 as pg
    fun = pg.PsfunDSerial()
    assert fun.set("VARIANT", variant) == 0 and fun.set("SCALING", float(scaling)) == 0
    return pg.PsfunDKrylov().apply(fun, pg.CsrMatrix.from_scipy(A), x, eps, itmax=m, istop=istop)


def check(lib, orc, A, x, m, scaling=-1.0, istop=2, variant="GENPADE"):
    orc.set_threads(0)
    g = solve(lib, A, x, m, scaling, istop, variant=variant)
    o = orc.krylov("ARNOLDI", orc.serial("EXP", variant, scaling), orc.Csr.from_scipy(A), x, 1e-10, itmax=m,
                   istop=istop)
    assert g.info == o["info"] and g.iter == o["iter"]
    if o["info"] == 0:
        assert np.linalg.norm(g.y - o["y"]) <= TOL * np.linalg.norm(o["y"])


def advection(n):
    """A banded nonsymmetric operator of norm ~4 with varying coefficients."""
    k = np.arange(n)
    return sp.diags([-1.0 - 0.3 * np.sin(k[1:]), 2.0 + 0.1 * np.cos(k), -0.7 * np.ones(max(n - 1, 0)),
                     0.2 * np.ones(max(n - 7, 0))][: 4 if n > 7 else 3], [-1, 0, 1, 7][: 4 if n > 7 else 3]).tocsr()


# rows: one block, a row group of 32 short or over by one row, 64 rows per
# block, the last block nearly empty, several rows per thread (524,287 rows:
# the largest size of this path); vectors: the smallest dimension, a pair, the
# largest basis in shared memory, one in global memory (64 x 20,000 rows fit,
# 128 x 40,000 do not)
@pytest.mark.parametrize("n,m", [(5, 3), (31, 4), (33, 8), (64, 2), (65, 12), (2049, 20), (9728, 64), (9729, 63),
                                 (20001, 64), (40000, 128), (97281, 24), (194561, 9), (524287, 8)])
def test_fixed_dimension(lib, orc, n, m):
    check(lib, orc, advection(n), np.random.default_rng(n).standard_normal(n), m)


@pytest.mark.parametrize("n,m", [(50, 20), (3000, 50), (70000, 64), (300001, 40)])
@pytest.mark.parametrize("variant", ["GENPADE", "CHBGEN"])
def test_to_a_tolerance(lib, orc, n, m, variant):
    check(lib, orc, advection(n), np.random.default_rng(n).standard_normal(n), m, istop=1, variant=variant)


def test_lost_orthogonality(lib):
    """Five distinct eigenvalues: the sixth vector is rounding noise and not
    orthogonal to the others, so the coefficients need the full substitution
    (psfun_d_arnoldi.f90:210-214 takes them one after another); the result is
    exp(A) x all the same."""
    d = np.repeat([-0.3, -1.1, -2.0, -2.9, -4.2], 700)
    x = np.random.default_rng(1).standard_normal(d.size)
    g = solve(lib, sp.diags(d).tocsr(), x, 14, scaling=1.0)
    y = np.exp(d) * x
    assert g.info == 0 and np.linalg.norm(g.y - y) <= TOL * np.linalg.norm(y)


@pytest.mark.parametrize("xs,As", [(1e-140, 1.0), (1e140, 1.0), (1.0, 1e-120), (1e100, 1e100), (1e-100, 1e-90)])
def test_extreme_scales(lib, orc, xs, As):
    """The windows follow the norms: x, and A with the scaling undoing it."""
    n = 3001
    check(lib, orc, As * advection(n), xs * np.random.default_rng(2).standard_normal(n), 16, scaling=-1.0 / As)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_input(lib, bad):
    x = np.ones(5000)
    x[4321] = bad
    g = solve(lib, advection(5000), x, 12)
    assert g.info != 0 or np.isnan(g.y).any()


def test_longest_row(lib, orc):
    """Rows of up to 64 entries take this path, one of 65 does not."""
    rng = np.random.default_rng(3)
    for longest in (64, 65):
        A = sp.random(4000, 4000, density=5 / 4000, random_state=4, format="lil")
        A[7] = 0.0
        A[7, rng.choice(4000, longest, replace=False)] = 0.05
        check(lib, orc, sp.csr_matrix(A), rng.standard_normal(4000), 30)
