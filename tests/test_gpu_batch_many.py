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
