"""GPU test of Householder factorizations whose levels run different kernels,
against the CPU oracle."""
import pytest

from alglin_b200 import bcr as B
from alglin_b200 import synth
from oracle import pyoracle as po
from tests._util import fwd_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nr,nx", [(6, 2, 2), (7, 0, 0), (8, 3, 3), (8, 0, 14), (10, 2, 2), (10, 2, 3), (10, 6, 6), (11, 0, 2),
                                     (11, 0, 3), (12, 0, 2), (12, 3, 3), (13, 5, 14), (16, 8, 16)])
@pytest.mark.parametrize("nblock", [9, 2400])
@pytest.mark.parametrize("select", ["QR", "QRP"])
@pytest.mark.parametrize("mixed", [False, True])
def test_levels_of_different_kernels(n, nr, nx, nblock, select, mixed):
    """Orders and columns on both sides of the lines between the register and the
    shared-memory kernel, with 1,200 pairs at the first level (just above the line for
    large levels) and few above; one pass and two.  Both solve to cond(A) * 2^-53;
    the oracle's own QR and LU solutions differ by at most 2e-13 here: bar 1e-9.
    The mixed path is refined to 1e-15."""
    qr, qx = max(0, nx - nr), max(0, nr - nx)
    s = synth.collocation(nblock, n, qr, qx, nr, nx, seed=n + nx)
    rhs = synth.rhs(s, 1, seed=n + 1)
    o = po.Oracle(s, select, "LU")
    assert o.factorize(), o.last_error()
    want = o.solve(rhs)
    h = B.BorderedCR()
    h.load_system(s)
    h.select(select)
    h.select_last("LU")
    if mixed:
        h.set_precision(B.PRECISION_MIXED)
        h.set_refinement(1e-15, 20)
    assert h.factorize(), h.last_error()
    x = rhs.copy()
    assert h.solve_n(1, x.reshape(-1), x.shape[1]), h.last_error()
    assert fwd_err(x[0, :s.ncols], want[0, :s.ncols]) < 1e-9
