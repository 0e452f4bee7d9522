"""BJAC on matrices whose diagonal blocks are tridiagonal, around the block
(32 rows) and block-group (1024 rows) sizes, and next to groups that are not."""
import numpy as np
import pytest
import scipy.sparse as sp

from psfun_gb300 import matrices

pytestmark = pytest.mark.gpu


def tridiagonal(n, seed):
    rng = np.random.default_rng(seed)
    e = -rng.uniform(0.2, 1.0, n - 1)
    e[rng.random(n - 1) < 0.1] = 0.0
    d = np.r_[0.0, -e] + np.r_[-e, 0.0] + rng.uniform(0.1, 1.0, n)
    return sp.csr_matrix(sp.diags([e, d, e], [-1, 0, 1]))


def cases():
    out = [(f"tri_{n}", tridiagonal(n, n)) for n in (2, 31, 32, 33, 1023, 1024, 1025, 1057, 5000)]
    out.append(("diagonal", sp.csr_matrix(sp.diags(np.linspace(1.0, 3.0, 1500)))))
    out.append(("grid_61", matrices.laplacian_2d(61)))
    # groups of both kinds in one matrix: narrow grid lines next to a tridiagonal part
    out.append(("mixed", sp.csr_matrix(sp.block_diag([tridiagonal(2100, 3), matrices.laplacian_2d(20),
                                                      tridiagonal(1300, 4)]))))
    return out


@pytest.mark.parametrize("name,A", cases(), ids=[c[0] for c in cases()])
def test_bjac_tridiagonal_blocks(lib, orc, name, A):
    import psfun_gb300 as pg
    n = A.shape[0]
    b = np.random.default_rng(5).standard_normal(n)
    x, info, it, err = pg.psb_krylov("CG", pg.CsrMatrix.from_scipy(A), "BJAC", b, 1.0, 0.1, np.zeros(n), 1e-12,
                                     itmax=3000, istop=2)
    o = orc.dcg(orc.Csr.from_scipy(A), b, 1.0, 0.1, eps=1e-12, itmax=3000, istop=2, prec="BJAC")
    assert info == 0 and o["info"] == 0 and err <= 1e-12
    assert abs(it - o["iter"]) <= 1
    # both residuals are below 1e-12 |b|, the smallest eigenvalue of A + 0.1 I is at least 0.1
    assert np.linalg.norm(x - o["x"]) <= 2 * 1e-12 * np.linalg.norm(b) / 0.1
