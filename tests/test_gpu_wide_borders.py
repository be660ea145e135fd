"""GPU tests of systems with many border rows, against the CPU oracle: sums over
the blocks of columns of 256 rows and more, and panels of more rows than the
blocked kernels take."""
import numpy as np
import pytest

from alglin_b200 import bcr as B
from alglin_b200 import synth
from oracle import pyoracle as po
from tests._util import fwd_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nx", [(255, 1), (256, 1), (257, 1), (300, 3), (512, 2), (513, 2), (600, 5)])
@pytest.mark.parametrize("nblock", [2, 9, 1500])
@pytest.mark.parametrize("select", ["LU", "QR"])
def test_columns_of_many_border_rows(nr, nx, nblock, select):
    """F's updates and the right-hand sides' border sums of columns that end just
    below, at and above one, two and three groups of 256 rows, over one block,
    several, and several parts; the product A x sums the same columns.  cond(A) is
    at most 4e2 at 2 and 9 blocks (dense SVD) and 6e7 at 1,500 (1-norm), which
    times 2^-53 gives 4e-14 and 7e-9: bars of 1e-11 and 1e-7."""
    bar = 1e-7 if nblock > 9 else 1e-11
    s = synth.dominant(nblock, 2, 0, nr - nx, nr, nx, seed=nr)
    # the border rows' pivots: the columns of Cq and F in turn
    for i in range(nr - nx):
        s.Cq[i, nx + i] += 10.0
    rhs = synth.rhs(s, 3, seed=nr + 1)
    o = po.Oracle(s, select, "LU")
    assert o.factorize(), o.last_error()
    want = o.solve(rhs)
    h = B.BorderedCR()
    h.load_system(s)
    h.select(select)
    h.select_last("LU")
    for fused in (False, True):
        x = rhs.copy()
        if fused:
            assert h.factorize_solve(3, x.reshape(-1), x.shape[1]), h.last_error()
        else:
            assert h.factorize(), h.last_error()
            assert h.solve_n(3, x.reshape(-1), x.shape[1]), h.last_error()
        for c in range(3):
            assert fwd_err(x[c, :s.ncols], want[c, :s.ncols]) < bar
    # A x: sums of at most nblock * n = 3,000 terms of one size
    ax, want = h.mv(rhs[0, :s.ncols]), o.mv(rhs[0, :s.ncols])
    assert np.abs(ax[:s.nrows] - want[:s.nrows]).max() <= 1e-11 * np.abs(want).max()


@pytest.mark.parametrize("n,nr,nx", [(128, 256, 1), (128, 257, 1), (100, 312, 20), (40, 432, 2), (33, 447, 2), (25, 463, 1)])
@pytest.mark.parametrize("nrhs", [1, 9])
def test_panels_of_about_512_rows(n, nr, nx, nrhs):
    """2n + nr = 512 rows, the most that the blocked FP64 kernel takes, and 513 and
    more, which run unblocked with factors L and M.  cond(A) <= 2e4 (dense SVD),
    2e4 * 2^-53 * 512 rows: 1e-9."""
    s = synth.collocation(3, n, 0, nr - nx, nr, nx, seed=n)
    for i in range(nr - nx):
        s.Cq[i, nx + i] += 10.0
    rhs = synth.rhs(s, nrhs, seed=n + 1)
    o = po.Oracle(s, "LU", "LU")
    assert o.factorize(), o.last_error()
    want = o.solve(rhs)
    h = B.BorderedCR()
    h.load_system(s)
    h.select("LU")
    h.select_last("LU")
    assert h.factorize(), h.last_error()
    x = rhs.copy()
    assert h.solve_n(nrhs, x.reshape(-1), x.shape[1]), h.last_error()
    for c in range(nrhs):
        assert fwd_err(x[c, :s.ncols], want[c, :s.ncols]) < 1e-9
