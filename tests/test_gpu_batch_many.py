"""Batched Lanczos with many instances, and its estimate monitors when a step
never comes."""
import time

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def test_monitor_wait_expires(lib, orc):
    """A monitor block whose step is never published gives up after the 2 s
    limit, all of its warps as one, with status 9002; the next batch works."""
    import torch

    import psfun_gb300 as pg
    from psfun_gb300 import matrices

    t0 = time.perf_counter()
    rc = lib.psfun_gpu_selftest_wait(2)
    dt = time.perf_counter() - t0
    assert rc == 9002, lib.psfun_gpu_last_error()
    assert 1.5 <= dt <= 30.0
    A = matrices.laplacian_2d(20)
    fun, meth = pg.PsfunDSerial(), pg.PsfunDKrylov()
    assert fun.set("VARIANT", "CHBSYM") == 0 and meth.set("KNAME", "LANCZOS") == 0
    x = np.random.default_rng(0).standard_normal((1, 400))
    X = torch.as_tensor(x, device="cuda")
    Y = torch.empty_like(X)
    _, infos, iters, _ = pg.krylov_batch(meth, fun, [(pg.CsrMatrix.from_scipy(A), X, Y, -0.5)], 1e-10, itmax=50,
                                         istop=1)
    o = orc.krylov("LANCZOS", orc.serial("EXP", "CHBSYM", 1.0), orc.Csr.from_scipy(sp.csr_matrix(-0.5 * A)), x[0],
                   1e-10, itmax=50, istop=1)
    assert not np.any(infos) and np.ravel(iters)[0] == o["iter"]
    assert np.linalg.norm(Y.cpu().numpy()[0] - o["y"]) <= 1e-10 * np.linalg.norm(o["y"])


@pytest.mark.parametrize("count,R,itmax,t,eps", [
    (130, 2, 60, -3.0, 1e-300),   # no pair converges: the step blocks are called in again and again
    (700, 1, 40, -3.0, 1e-300),   # more estimates per step than warps
    (3, 4, 330, -40.0, 1e-300),   # few instances, high orders: the lag of few monitors
    (257, 3, 50, -1.0, 1e-8),     # pairs end at different steps while estimates are handed over
    (1, 1, 400, -60.0, 1e-12),
])
def test_estimates_handed_to_the_steps(lib, count, R, itmax, t, eps):
    """Every pair ends where the same solve alone ends, with its result and its
    error estimate, whoever has done its estimates."""
    import torch

    import psfun_gb300 as pg
    from psfun_gb300 import matrices

    fun, meth, single = pg.PsfunDSerial(), pg.PsfunDKrylov(), pg.PsfunDKrylov()
    assert fun.set("VARIANT", "CHBSYM") == 0
    assert meth.set("KNAME", "LANCZOS") == 0 and single.set("KNAME", "LANCZOS") == 0
    items = []
    for k in range(count):
        A = matrices.laplacian_2d(19 + k % 7)
        X = torch.as_tensor(np.random.default_rng(k).standard_normal((R, A.shape[0])), device="cuda")
        items.append((A, pg.CsrMatrix.from_scipy(sp.csr_matrix(A)), X, torch.empty_like(X),
                      t * (0.4 + 0.6 * (k % 5) / 5)))
    _, infos, iters, errs = pg.krylov_batch(meth, fun, [i[1:] for i in items], eps, itmax=itmax, istop=1)
    infos, iters, errs = (np.reshape(v, (count, R)) for v in (infos, iters, errs))
    assert not infos.any()
    for k in sorted({0, 1, count // 2, count - 1} & set(range(count))):
        A, _, X, Y, tk = items[k]
        a = pg.CsrMatrix.from_scipy(sp.csr_matrix(tk * A))
        for q in range(R):
            r = single.apply(fun, a, X[q].clone(), eps, itmax=itmax, istop=1)
            assert r.info == 0 and iters[k, q] == r.iter
            # f(H) is bounded by 1; both bases carry O(m eps) rounding
            tol = 200 * itmax * np.finfo(float).eps * float(torch.linalg.norm(X[q]))
            assert float((Y[q] - r.y).abs().max()) <= tol
            assert errs[k, q] <= max(10 * r.err, 1e-12)


def test_many_instances_without_convergence(lib):
    """3000 instances, 199 estimates each that do not converge: more work than
    the bounded wait at the end of the steps would sit out if it were left to
    the monitors (~2.2 s against 2 s)."""
    import torch

    import psfun_gb300 as pg
    from psfun_gb300 import matrices

    fun, meth, single = pg.PsfunDSerial(), pg.PsfunDKrylov(), pg.PsfunDKrylov()
    assert fun.set("VARIANT", "CHBSYM") == 0
    assert meth.set("KNAME", "LANCZOS") == 0 and single.set("KNAME", "LANCZOS") == 0
    A = [matrices.laplacian_2d(18 + k) for k in range(4)]
    h = [pg.CsrMatrix.from_scipy(sp.csr_matrix(a)) for a in A]
    X = [torch.as_tensor(np.random.default_rng(k).standard_normal((1, a.shape[0])), device="cuda")
         for k, a in enumerate(A)]
    items = [(h[k % 4], X[k % 4], torch.empty_like(X[k % 4]), -3.0) for k in range(3000)]
    info, infos, iters, _ = pg.krylov_batch(meth, fun, items, 1e-300, itmax=200, istop=1)
    assert info == 0 and not np.any(infos)
    for k in (0, 1500, 2999):
        a = pg.CsrMatrix.from_scipy(sp.csr_matrix(-3.0 * A[k % 4]))
        r = single.apply(fun, a, X[k % 4][0].clone(), 1e-300, itmax=200, istop=1)
        assert r.info == 0 and iters[k, 0] == r.iter
        tol = 200 * 200 * np.finfo(float).eps * float(torch.linalg.norm(X[k % 4]))
        assert float((items[k][2][0] - r.y).abs().max()) <= tol
