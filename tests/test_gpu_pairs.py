"""GPU tests of the pair kernels at the sizes and values where they can go
wrong, against the CPU oracle.

Bar: forward error against the oracle's solution <= 1e-10, the bar of the other
parity tests.  Both sides solve the same system backward stably, so they differ
by cond(A) * 2^-53 times a modest power of n; cond(A) of these systems is at
most 6e3 (dense SVD), which gives 7e-13 times that power."""
import numpy as np
import pytest

from alglin_b200 import bcr as B
from alglin_b200 import synth
from oracle import pyoracle as po
from tests._util import fwd_err

pytestmark = pytest.mark.gpu


def solve_both(s, rhs, select="LU"):
    """Solutions of the library (factorize, then solve), of the library in one
    factorize + solve, and of the oracle."""
    o = po.Oracle(s, select, "LU")
    assert o.factorize(), o.last_error()
    xo = o.solve(rhs)
    out = []
    for fused in (False, True):
        h = B.BorderedCR()
        h.load_system(s)
        h.select(select)
        h.select_last("LU")
        x = rhs.copy()
        if fused:
            assert h.factorize_solve(x.shape[0], x.reshape(-1), x.shape[1]), h.last_error()
        else:
            assert h.factorize(), h.last_error()
            assert h.solve_n(x.shape[0], x.reshape(-1), x.shape[1]), h.last_error()
        out.append(x)
    return out[0], out[1], xo


def check(s, rhs, select="LU", bar=1e-10):
    x1, x2, xo = solve_both(s, rhs, select)
    for x in (x1, x2):
        for c in range(rhs.shape[0]):
            assert fwd_err(x[c, :s.ncols], xo[c, :s.ncols]) < bar


@pytest.mark.parametrize("n", [8, 16])
@pytest.mark.parametrize("exponent", [0, -1021, 1010])
def test_pivots_of_every_magnitude(n, exponent):
    """Block rows scaled by 2^exponent, to about the ends of the range in which the
    oracle itself stays finite.  At 2^-1021 the intermediate values are rounded
    to 2^-53 of the entries at worst, so the bar stands."""
    s = synth.collocation(37, n, 1, 1, 3, 3, seed=5)
    for a in (s.D, s.E, s.B):
        np.ldexp(a, exponent, out=a)
    rhs = synth.rhs(s, 2, seed=6)
    rhs[:, :s.n * s.nblock] = np.ldexp(rhs[:, :s.n * s.nblock], exponent)
    check(s, rhs)


@pytest.mark.parametrize("n", [8, 16])
@pytest.mark.parametrize("nblock", [2, 3, 33])
def test_pivot_ties_follow_getrf(n, nblock):
    """Entries of +-1 and +-1/2 only: many candidates of exactly equal
    magnitude, where getrf takes the first position.  The oracle applies that
    rule, so a different choice would show as another rounding, not as an
    error; cond(A) <= 2e4 here, so the bar is 1e-8, whichever row wins."""
    s = synth.dominant(nblock, n, 0, 0, 2, 2, seed=3)
    rng = np.random.default_rng(7)
    s.D[:] = rng.choice([-1.0, -0.5, 0.5, 1.0], s.D.shape)
    s.E[:] = rng.choice([-1.0, -0.5, 0.5, 1.0], s.E.shape)
    check(s, synth.rhs(s, 1, seed=8), bar=1e-8)


@pytest.mark.parametrize("n,nr,nx", [(25, 0, 0), (32, 9, 9), (33, 1, 2), (40, 3, 3), (63, 5, 5), (64, 8, 8), (65, 2, 2),
                                     (72, 0, 0), (100, 17, 17), (127, 4, 4), (128, 16, 16)])
@pytest.mark.parametrize("nblock", [2, 3, 37])
def test_large_block_lu(n, nr, nx, nblock):
    """The blocked FP64 kernel at the edges of its tiles: block widths that are no
    multiple of 8 or 16, one and two panel blocks, no borders and borders that
    pass a tile, one pair (columns split over a cluster) and many.  cond(A) is at
    most 3e4 here (dense SVD), so the bar is 1e-9: 3e4 * 2^-53 * 256 rows."""
    qx = max(0, nr - nx)
    qr = max(0, nx - nr)
    s = synth.collocation(nblock, n, qr, qx, nr, nx, seed=n)
    check(s, synth.rhs(s, 3, seed=n + 1), bar=1e-9)


@pytest.mark.parametrize("n", [17, 31, 32, 33, 64, 65, 127, 128])
@pytest.mark.parametrize("nrhs", [1, 8, 9, 17])
@pytest.mark.parametrize("mode", ["LU", "QRP", "mixed"])
def test_large_block_sweeps(n, nrhs, mode):
    """The sweeps for n > 16 at the edges of their runs of 32 columns, of the row
    counts their threads are built for and of the chunks of right-hand sides
    (8, after the 16 of a solve), with L and M, with the operator form and with
    QRP's column map.  Bar: as test_large_block_lu; the mixed path is refined to
    1e-15 relative residual, which cond(A) <= 3e4 turns into 3e-11."""
    s = synth.collocation(5, n, 0, 0, 3, 3, seed=n)
    rhs = synth.rhs(s, nrhs, seed=n + 1)
    if mode != "mixed":
        return check(s, rhs, mode, bar=1e-9)
    o = po.Oracle(s, "LU", "LU")
    assert o.factorize(), o.last_error()
    xo = o.solve(rhs)
    h = B.BorderedCR()
    h.load_system(s)
    h.set_precision(B.PRECISION_MIXED)
    h.set_refinement(1e-15, 10)
    assert h.factorize(), h.last_error()
    x = rhs.copy()
    assert h.solve_n(nrhs, x.reshape(-1), x.shape[1]), h.last_error()
    assert h.refinement_info()[1] <= 1e-15
    for c in range(nrhs):
        assert fwd_err(x[c, :s.ncols], xo[c, :s.ncols]) < 1e-9


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 15, 16])
@pytest.mark.parametrize("nr,nx", [(0, 0), (1, 3), (8, 8), (5, 16)])
@pytest.mark.parametrize("select", ["QR", "QRP"])
def test_qr_panels(n, nr, nx, select):
    """The warp QR kernel from one column to a full warp of rows, with all columns
    in one pass and in two, and its column map.  cond(A) <= 6e3 (dense SVD)."""
    s = synth.collocation(9, n, max(0, nx - nr), max(0, nr - nx), nr, nx, seed=n)
    check(s, synth.rhs(s, 2, seed=n + 1), select, bar=1e-9)


@pytest.mark.parametrize("select", ["QR", "QRP"])
def test_qr_zero_column_is_reported(select):
    """A panel column that is zero in both its row blocks: R has a zero on its
    diagonal, the factorization fails, and the library stays usable."""
    s = synth.collocation(6, 7, 0, 0, 2, 2, seed=3)
    bad = s.copy()
    bad.E[2, 4] = 0.0  # column 4 of E_2 and D_3 (stored by columns)
    bad.D[3, 4] = 0.0
    h = B.BorderedCR()
    h.load_system(bad)
    h.select(select)
    assert not h.factorize()
    check(s, synth.rhs(s, 1, seed=4), select)


@pytest.mark.parametrize("n", [1, 4, 5, 7, 9, 12, 15])
@pytest.mark.parametrize("nr,nx", [(0, 0), (3, 4), (8, 8)])
@pytest.mark.parametrize("nblock", [2, 3, 40])
def test_padded_warp_lu(n, nr, nx, nblock):
    """Orders between the warp kernel's 8 and 16, as leading parts of such blocks:
    factorize + solve with the right-hand sides in the factorization (up to 8 - nx)
    and apart from it.  cond(A) <= 4e4 (dense SVD)."""
    s = synth.collocation(nblock, n, max(0, nx - nr), max(0, nr - nx), nr, nx, seed=n)
    check(s, synth.rhs(s, 4, seed=n + 1), bar=1e-9)
    if nr + max(0, nx - nr) == nx + max(0, nr - nx):
        rhs = synth.rhs(s, 1, seed=n + 2)
        o = po.Oracle(s, "LU", "LU")
        assert o.factorize(), o.last_error()
        h = B.BorderedCR()
        h.load_system(s)
        h.set_precision(B.PRECISION_MIXED)
        h.set_refinement(1e-15, 10)
        x = rhs.copy()
        assert h.factorize_solve(1, x.reshape(-1), x.shape[1]), h.last_error()
        assert fwd_err(x[0, :s.ncols], o.solve(rhs)[0, :s.ncols]) < 1e-9


@pytest.mark.parametrize("n", [17, 24, 31, 32])
@pytest.mark.parametrize("nr,nx", [(0, 0), (1, 8), (8, 2)])
@pytest.mark.parametrize("nblock", [2, 29])
def test_padded_cta_lu(n, nr, nx, nblock):
    """Orders between 16 and 32 as leading parts of the CTA kernel's blocks.
    cond(A) <= 2e5 (dense SVD), 2e5 * 2^-53 * 64 rows."""
    s = synth.collocation(nblock, n, max(0, nx - nr), max(0, nr - nx), nr, nx, seed=n)
    check(s, synth.rhs(s, 5, seed=n + 1), bar=1e-9)


@pytest.mark.parametrize("n", [12, 20, 32])
def test_zero_pivot_in_the_warp_and_cta_kernels(n):
    """A zero column in both row blocks of a pair: getrf's INFO, and the handle's
    next matrix is factored correctly."""
    s = synth.collocation(6, n, 0, 0, 2, 2, seed=3)
    bad = s.copy()
    bad.E[2, 5] = 0.0
    bad.D[3, 5] = 0.0
    h = B.BorderedCR()
    h.load_system(bad)
    h.select("LU")
    assert not h.factorize()
    assert "INFO = 6" in h.last_error()
    h.load_system(s)
    assert h.factorize(), h.last_error()
    check(s, synth.rhs(s, 1, seed=4))


@pytest.mark.parametrize("n", [8, 16])
@pytest.mark.parametrize("nrhs", [2, 7, 8, 9, 17])
@pytest.mark.parametrize("nblock,nr,nx", [(1, 0, 0), (2, 1, 3), (37, 5, 4), (200, 8, 8)])
@pytest.mark.parametrize("select", ["LU", "QR", "QRP"])
def test_sweeps_of_several_right_hand_sides(n, nrhs, nblock, nr, nx, select):
    """The sweeps that take eight right-hand sides of a pair at once: a part of a
    chunk, a whole one, a remainder of one; borders of zero, of less than the
    products' four columns, and of eight.  cond(A) <= 6e3 (dense SVD)."""
    s = synth.collocation(nblock, n, max(0, nx - nr), max(0, nr - nx), nr, nx, seed=n)
    check(s, synth.rhs(s, nrhs, seed=n + 1), select)


@pytest.mark.parametrize("n", [33, 40, 95, 128])
@pytest.mark.parametrize("nblock,nr,nx", [(2, 0, 0), (3, 1, 1), (40, 16, 16), (5, 13, 4)])
def test_large_block_fp32_panels(n, nblock, nr, nx):
    """The tensor-core pair kernel's panel with a partial last block, border rows
    in a warp of their own and in one with pivot rows, and its products with no
    borders and the most.  Bar: test_large_block_sweeps' for the mixed path."""
    s = synth.collocation(nblock, n, max(0, nx - nr), max(0, nr - nx), nr, nx, seed=n)
    rhs = synth.rhs(s, 2, seed=n + 1)
    o = po.Oracle(s, "LU", "LU")
    assert o.factorize(), o.last_error()
    xo = o.solve(rhs)
    h = B.BorderedCR()
    h.load_system(s)
    h.set_precision(B.PRECISION_MIXED)
    h.set_refinement(1e-15, 10)
    assert h.factorize(), h.last_error()
    x = rhs.copy()
    assert h.solve_n(2, x.reshape(-1), x.shape[1]), h.last_error()
    for c in range(2):
        assert fwd_err(x[c, :s.ncols], xo[c, :s.ncols]) < 1e-9
