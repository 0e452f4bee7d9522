"""Batched Lanczos whose estimates run beside the steps: every pair ends at the
iteration at which the same solve alone ends, whatever the number of
instances per estimate warp, and next to pairs that end by breakdown, by a
zero right-hand side or at itmax."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def instance(pg, matrices, kind, seed, R):
    rng = np.random.default_rng(seed)
    if kind == "identity":  # every pair breaks down after one step (exactly: a coordinate vector)
        return sp.identity(37, format="csr"), np.eye(37)[:R], -0.5
    A = matrices.laplacian_2d(8 + seed % 29)
    X = rng.standard_normal((R, A.shape[0]))
    if kind == "zero":
        X[0] = 0.0
    t = {"slow": -6.0}.get(kind, -0.05 - 0.09 * (seed % 11))
    return sp.csr_matrix(A), X, t


@pytest.mark.parametrize("count,R,itmax", [(1, 1, 2), (1, 4, 40), (2, 3, 5), (3, 2, 25), (24, 4, 40), (90, 2, 30)])
def test_pairs_end_where_the_single_solve_does(lib, count, R, itmax):
    import psfun_gb300 as pg
    from psfun_gb300 import matrices

    kinds = ["plain"] if count == 1 else ["plain", "slow", "identity", "plain", "zero"]
    fun, meth = pg.PsfunDSerial(), pg.PsfunDKrylov()
    fun.set("VARIANT", "CHBSYM")
    meth.set("KNAME", "LANCZOS")
    data = [instance(pg, matrices, kinds[k % len(kinds)], k, R) for k in range(count)]
    items, handles = [], []
    for A, X, t in data:
        h = pg.CsrMatrix.from_scipy(A)
        x = torch.as_tensor(X, device="cuda")
        handles.append(h)
        items.append((h, x, torch.empty_like(x), t))
    eps = 1e-8
    _, infos, iters, _ = pg.krylov_batch(meth, fun, items, eps, itmax=itmax, istop=1)
    infos, iters = np.reshape(infos, (count, R)), np.reshape(iters, (count, R))
    for k, (A, X, t) in enumerate(data):
        single = pg.PsfunDKrylov()
        single.set("KNAME", "LANCZOS")
        tA = pg.CsrMatrix.from_scipy(sp.csr_matrix(t * A))
        got = items[k][2].cpu().numpy()
        for q in range(R):
            if not X[q].any():
                assert iters[k, q] == 0 and not got[q].any()
                continue
            if infos[k, q]:
                # a projected matrix that is empty: breakdown at the first step, or itmax = 2
                assert itmax == 2 or kinds[k % len(kinds)] == "identity"
                continue
            r = single.apply(fun, tA, torch.as_tensor(X[q], device="cuda"), eps, itmax=itmax, istop=1)
            assert r.iter == iters[k, q]
            # both bases carry O(m eps) rounding, f(H) is bounded by 1
            assert np.abs(got[q] - r.y.cpu().numpy()).max() <= 200 * itmax * EPS * np.linalg.norm(X[q])
