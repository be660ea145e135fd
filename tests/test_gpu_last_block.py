"""GPU tests of last blocks of every size, against the CPU oracle or a solution
that is known."""
import numpy as np
import pytest

from alglin_b200 import bcr as B
from alglin_b200 import synth
from oracle import pyoracle as po
from tests._util import fwd_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [960, 961, 976, 977, 1100])
@pytest.mark.parametrize("last", ["LU", "QR"])
@pytest.mark.parametrize("batch", [False, True])
def test_last_blocks_of_about_a_thousand_rows(order, last, batch):
    """Last blocks whose two work vectors do not fit in what a kernel may use of
    shared memory without asking (orders of 961 and above).  cond(A) <= 3e3 (dense
    SVD), 3e3 * 2^-53 * 1,100 rows = 4e-10: bar 1e-9."""
    n = 4
    q = order - 2 * n
    s = synth.collocation(5, n, q, q, 0, 0, seed=order)
    for i in range(q):
        s.H[2 * n + i, n + i] += 40.0
    rhs = synth.rhs(s, 1, seed=3)
    o = po.Oracle(s, "LU", last)
    assert o.factorize(), o.last_error()
    want = o.solve(rhs)
    h = B.BorderedCR()
    h.load_system(s)
    h.select("LU")
    h.select_last(last)
    x = rhs.copy()
    if batch:
        bt = B.Batch([h])
        bt.prepare()
        assert bt.factorize(), bt.last_error()
        xs = [x[0]]
        assert bt.solve(xs), bt.last_error()
        x = np.array(xs)
    else:
        assert h.factorize(), h.last_error()
        assert h.solve_n(1, x.reshape(-1), x.shape[1]), h.last_error()
    assert fwd_err(x[0, :s.ncols], want[0, :s.ncols]) < 1e-9


def test_a_launch_that_does_not_fit_is_an_error():
    """A last block whose two work vectors are larger than an SM's shared memory: the
    launch of its solve is refused, and the call says so.  (The matrix is zero, so
    that its factorization ends at the first pivot.)  The handle stays usable."""
    h = B.BorderedCR()
    h.allocate(1, 2, 12600, 12600, 0, 0)
    x = np.zeros(h.ncols())
    with pytest.raises(B.BCRError, match="launch"):
        h.factorize_solve(1, x, x.size)
    s = synth.collocation(5, 4, 0, 0, 2, 2, seed=1)
    rhs = synth.rhs(s, 1, seed=3)
    o = po.Oracle(s, "LU", "LU")
    assert o.factorize(), o.last_error()
    h.load_system(s)
    x = rhs.copy()
    assert h.factorize_solve(1, x.reshape(-1), x.shape[1]), h.last_error()
    # cond(A) = 19 (dense SVD)
    assert fwd_err(x[0, :s.ncols], o.solve(rhs)[0, :s.ncols]) < 1e-12


@pytest.mark.parametrize("n", [2, 8, 16, 32, 33, 128])
@pytest.mark.parametrize("nrhs", [1, 3])
@pytest.mark.parametrize("batch", [False, True])
def test_last_pivot_below_the_normal_numbers(n, nrhs, batch):
    """A single block, so that the last block is the matrix, of order 4 to 256, whose
    last pivot is 2^-1026: its reciprocal overflows, the quotients do not.  The
    last row has no other element and its unknown is a small integer, so that its
    right-hand side and the quotient are exact."""
    if batch and (n > 32 or n == 2 or nrhs > 1):
        pytest.skip("batches take one right-hand side and their own block orders")
    N, tiny = 2 * n, np.ldexp(1.0, -1026)
    rng = np.random.default_rng(n)
    A = rng.standard_normal((N, N)) * 0.1 + 4.0 * np.eye(N)
    A[-1] = 0.0
    A[-1, -1] = tiny
    s = synth.collocation(1, n)
    s.D[0], s.E[0] = A[:n, :n].T, A[:n, n:].T
    s.H[:] = A[n:].T
    want = rng.standard_normal((nrhs, N))
    want[:, -1] = rng.integers(1, 8, nrhs)
    x = want @ A.T
    x[:, -1] = want[:, -1] * tiny
    assert (x[:, -1] / tiny == want[:, -1]).all()
    h = B.BorderedCR()
    h.load_system(s)
    h.select("LU")
    h.select_last("LU")
    if batch:
        bt = B.Batch([h])
        bt.prepare()
        assert bt.factorize(), bt.last_error()
        xs = [x[0].copy()]
        assert bt.solve(xs), bt.last_error()
        x = np.array(xs)
    else:
        assert h.factorize(), h.last_error()
        assert h.solve_n(nrhs, x.reshape(-1), x.shape[1]), h.last_error()
    assert (x[:, -1] == want[:, -1]).all()
    assert np.abs(x - want).max() < 1e-12 * np.abs(want).max()
