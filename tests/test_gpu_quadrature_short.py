"""Quadrature sums whose Krylov space ends after one, two, three or a few
steps (as many as the matrix has distinct eigenvalues): the elimination beside
the steps has then done no row, the first, or all but the last."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distinct", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("itmax", [1, 2, 3, 50])
def test_short_spaces(lib, distinct, itmax):
    torch = pytest.importorskip("torch")
    import psfun_gb300 as pg
    n = 700
    lam = 1.0 + np.arange(n) % distinct / 8.0  # in [1, 1.75]
    a = pg.CsrMatrix.from_scipy(sp.csr_matrix(sp.diags(lam)))
    q = pg.PsfunZQuadrature()
    q.computepoles(pg.hhtmethod1, lambda z: 1.0 / np.sqrt(z), 16, rparams=[0.9, 2.0])
    q.setmatrix(a)
    x = np.random.default_rng(distinct).standard_normal(n)
    y = torch.empty(n, dtype=torch.float64, device="cuda")
    y, info, it, _ = q.apply(torch.tensor(x, device="cuda"), eps=1e-13, itmax=itmax, y=y)
    assert info == 0 and 1 <= it <= itmax
    if itmax >= distinct:
        # the rule's error for 16 poles on [0.9, 2] is far below 1e-10
        assert np.abs(y.cpu().numpy() - x / np.sqrt(lam)).max() <= 1e-10 * np.abs(x).max()
