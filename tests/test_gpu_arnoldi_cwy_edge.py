"""Arnoldi solves to a tolerance next to 2^19 rows, where the estimate monitors
leave the fewest blocks to the steps and a warp's row group is the widest:
every row has to enter the dots."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


# 522,240 rows: the last size with six rows per lane on 136 blocks; 522,241:
# the first with seven; 524,287: the largest size of this path
@pytest.mark.parametrize("n", [522240, 522241, 524287])
@pytest.mark.parametrize("start", ["random", "row"])
def test_every_row_enters_the_dots(lib, orc, n, start):
    import psfun_gb300 as pg
    k = np.arange(n)
    A = sp.diags([-1.0 - 0.3 * np.sin(k[1:]), 2.0 + 0.1 * np.cos(k), -0.7 * np.ones(n - 1), 0.2 * np.ones(n - 7)],
                 [-1, 0, 1, 7]).tocsr()
    x = np.random.default_rng(n).standard_normal(n) if start == "random" else (k == 200).astype(float)
    orc.set_threads(0)
    fun = pg.PsfunDSerial()
    assert fun.set("VARIANT", "GENPADE") == 0 and fun.set("SCALING", -3.0) == 0
    g = pg.PsfunDKrylov().apply(fun, pg.CsrMatrix.from_scipy(A), x, 1e-10, itmax=60, istop=1)
    o = orc.krylov("ARNOLDI", orc.serial("EXP", "GENPADE", -3.0), orc.Csr.from_scipy(A), x, 1e-10, itmax=60, istop=1)
    assert g.info == 0 and o["info"] == 0 and g.iter == o["iter"]
    # both reach the tolerance 1e-10 in the same space: equal up to rounding, as for every Krylov result here
    assert np.linalg.norm(g.y - o["y"]) <= 1e-10 * np.linalg.norm(o["y"])
