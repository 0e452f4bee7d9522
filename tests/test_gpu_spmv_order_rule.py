"""Whether a handle takes the rows of its tiles by length depends on the matrix
alone, not on how many host threads counted: next to the line (the plain
schedule 1.25 times the entries' instructions) the product has the bits of the
side on which the whole groups of 32 rows put it."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


# 4100 groups of 32 rows of 3 entries, some of which hold a row of 24.  With 152
# of those the plain schedule is half a group below the line, with 153 above; a
# group that a cut between threads splits would count for one more.
@pytest.mark.parametrize("long_rows,by_length", [(152, False), (153, True)])
def test_next_to_the_line(lib, long_rows, by_length):
    torch = pytest.importorskip("torch")
    import psfun_gb300 as pg
    n = 131200
    lens = np.full(n, 3)
    at = 32 * 26 * np.arange(long_rows) + 5
    lens[at] = 24
    irp = np.r_[0, np.cumsum(lens)]
    rng = np.random.default_rng(1)
    ja = np.repeat(rng.integers(0, n - 200, n), lens) + (np.arange(irp[-1]) - np.repeat(irp[:-1], lens)) * 7
    val = rng.standard_normal(irp[-1])
    x = rng.choice([-1.0, 1.0], n)  # exact products
    a = pg.CsrMatrix.from_scipy(sp.csr_matrix((val, ja, irp), shape=(n, n)))
    y = a.spmv(torch.as_tensor(x, device="cuda")).cpu().numpy()
    p = (val * x[ja])[irp[at][:, None] + np.arange(24)]  # the long rows' products
    plain, two = np.zeros(long_rows), np.zeros((2, long_rows))
    for k in range(24):  # one sum in order; two sums that take the eights in turn
        plain += p[:, k]
        two[(k // 8) % 2] += p[:, k]
    want = two[0] + two[1] if by_length else plain
    assert not np.array_equal(plain, two[0] + two[1])
    assert np.array_equal(y[at], want)
