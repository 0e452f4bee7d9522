"""Handles made, solved with and deleted in turn by one method object: the same
sizes get the same device addresses again, and nothing of the matrix that is
gone may act on the next one."""
import numpy as np
import pytest

from psfun_gb300 import matrices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kname,variant", [("LANCZOS", "CHBSYM"), ("ARNOLDI", "GENPADE")])
@pytest.mark.parametrize("istop", [1, 2])
def test_norms_of_very_different_size(lib, orc, kname, variant, istop):
    import psfun_gb300 as pg
    L = matrices.laplacian_2d(150)
    x = np.random.default_rng(1).standard_normal(L.shape[0])
    fun, meth = pg.PsfunDSerial(), pg.PsfunDKrylov()
    assert fun.set("VARIANT", variant) == 0 and meth.set("KNAME", kname) == 0
    y = np.empty_like(x)
    for scale in 3 * (1e-6, 1.0, 1e-9, 1e-2):
        A = -scale * L
        a = pg.CsrMatrix.from_scipy(A)
        r = meth.apply(fun, a, x, 1e-10, itmax=40, istop=istop, y=y)
        del a
        o = orc.krylov(kname, orc.serial("EXP", variant, 1.0), orc.Csr.from_scipy(A), x, 1e-10, itmax=40, istop=istop)
        assert r.info == 0 and o["info"] == 0 and r.iter == o["iter"]
        assert np.linalg.norm(r.y - o["y"]) <= 1e-10 * np.linalg.norm(o["y"])
