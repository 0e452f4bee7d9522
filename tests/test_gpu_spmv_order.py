"""The product on rows of very different length, where the rows of a tile are
taken by descending length: tiles of one row, of 480 and of the rows left
over, empty rows, rows around the warp split and longer than a tile."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def matrix(lens, seed):
    rng = np.random.default_rng(seed)
    n = len(lens)
    indptr = np.r_[0, np.cumsum(lens)]
    cols = np.concatenate([np.sort(rng.choice(n, l, replace=False)) for l in lens]) if n else np.zeros(0)
    return sp.csr_matrix((rng.standard_normal(indptr[-1]), cols.astype(np.int32), indptr), shape=(n, n))


def lengths(name):
    rng = np.random.default_rng(len(name))
    if name == "sparse_tiles":  # full tiles of 480 rows, most of them empty or short
        l = rng.integers(0, 3, 20000)
        l[::61] = 200
    elif name == "rest":  # a last tile of few rows
        l = np.where(np.arange(480 * 30 + 7) % 33 == 0, 120, 2)
    elif name == "split":  # around the threshold of the warp split
        l = rng.choice([1, 31, 32, 33, 40, 63, 64, 65, 300], 3001)
    elif name == "longer_than_tile":
        l = rng.choice([1, 5, 90], 6000)
        l[[0, 7, 2999, 5999]] = [4095, 4096, 4097, 5900]
    else:  # power law
        l = np.minimum(4.0 * rng.random(30001) ** (-1.0 / 1.5), 4000).astype(int)
    return l


@pytest.mark.parametrize("name", ["sparse_tiles", "rest", "split", "longer_than_tile", "power"])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_rows_by_length(lib, name, beta):
    torch = pytest.importorskip("torch")
    import psfun_gb300 as pg
    A = matrix(lengths(name), 3)
    n = A.shape[0]
    rng = np.random.default_rng(4)
    x, y0 = rng.standard_normal(n), rng.standard_normal(n)
    y = torch.tensor(y0, device="cuda")
    pg.CsrMatrix.from_scipy(A).spmv(torch.tensor(x, device="cuda"), alpha=1.5, beta=beta, y=y)
    want = 1.5 * (A @ x) + beta * y0
    # each side adds the row's products in some order: len eps sum |a x| each, and the last operations
    bound = 1.5 * (abs(A) @ abs(x))
    tol = (2 * np.diff(A.indptr) + 8) * EPS * (bound + abs(beta * y0))
    assert (np.abs(y.cpu().numpy() - want) <= tol).all()
