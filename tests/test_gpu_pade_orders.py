"""GENPADE and phi through the serial entry at the edges of the evaluation: the
Pade approximant below degree 6 and the Taylor polynomial from 6 on, orders
around the shared-memory and group limits, and norms with no, one, two and many
squarings (a single block replaces the last two by products with the vector).
Against the oracle's DGPADM, 1e-11 relative as for every dense f(H) here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-11


def check(orc, H, x, degree, fname="EXP", phiorder=1):
    import psfun_gb300 as pg
    f = pg.PsfunDSerial()
    assert f.set("FNAME", fname) == 0 and f.set("VARIANT", "GENPADE") == 0
    assert f.set("PADE_DEGREE", degree) == 0 and f.set("PHIORDER", phiorder) == 0
    y, info = f.apply(H, x)
    o = orc.serial(fname, "GENPADE", 1.0, padedegree=degree, phiorder=phiorder)
    yo, infoo = orc.serial_apply(o, H, x)
    assert info == infoo == 0
    assert np.linalg.norm(y - yo) <= TOL * np.linalg.norm(yo)


def matrix(m, norm, seed):
    rng = np.random.default_rng(seed)
    H = rng.standard_normal((m, m)) - 2.0 * np.eye(m)
    return H * (norm / np.abs(H).sum(axis=1).max()), rng.standard_normal(m)


@pytest.mark.parametrize("m", [1, 2, 3, 19, 20, 27, 28, 29, 33, 80, 129])
@pytest.mark.parametrize("degree", [5, 6, 9])
def test_orders(lib, orc, m, degree):
    check(orc, *matrix(m, 7.3, m), degree)


@pytest.mark.parametrize("norm", [0.03, 0.4, 0.5, 0.6, 1.0, 1.9, 2.0, 4.0, 8.0, 30.0])
@pytest.mark.parametrize("m", [6, 34])
def test_norms(lib, orc, norm, m):
    check(orc, *matrix(m, norm, 5), 6)


@pytest.mark.parametrize("m", [1, 17, 26, 27, 45])
@pytest.mark.parametrize("phiorder", [1, 2, 4])
def test_phi(lib, orc, m, phiorder):
    check(orc, *matrix(m, 3.1, m), 6, "PHI", phiorder)
