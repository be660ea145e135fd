"""GPU tests of pivots and columns at the ends of the floating-point range.

The columns of chosen unknowns are scaled by powers of two, which changes no
pivot, no multiplier and no rounding as long as nothing leaves the range: the
solution is that of the unscaled system with those unknowns scaled back, which
the CPU oracle gives."""
import numpy as np
import pytest

from alglin_b200 import bcr as B
from alglin_b200 import synth
from oracle import pyoracle as po
from tests._util import fwd_err

pytestmark = pytest.mark.gpu


def scale_unknown(s, k, c, e):
    """Column c of block unknown x_k times 2^e."""
    if k < s.nblock:
        s.D[k, c] = np.ldexp(s.D[k, c], e)
    if k > 0:
        s.E[k - 1, c] = np.ldexp(s.E[k - 1, c], e)
    s.C[k, c] = np.ldexp(s.C[k, c], e)
    if k == 0:
        s.H[c] = np.ldexp(s.H[c], e)
    if k == s.nblock:
        s.H[s.n + c] = np.ldexp(s.H[s.n + c], e)


def scaled_system(n, nblock, scales, seed):
    """The system with unknown (k, c) scaled by 2^scales[k, c], right-hand sides of
    moderate size and the unscaled solution."""
    s = synth.collocation(nblock, n, 0, 0, 2, 2, seed=seed)
    rhs = np.ldexp(synth.rhs(s, 2, seed=seed + 1), -10)
    o = po.Oracle(s, "LU", "LU")
    assert o.factorize(), o.last_error()
    want = o.solve(rhs)
    t = s.copy()
    for (k, c), e in scales.items():
        scale_unknown(t, k, c, e)
    return t, rhs, want


def unscale(s, x, scales):
    y = x.copy()
    for (k, c), e in scales.items():
        y[:, k * s.n + c] = np.ldexp(y[:, k * s.n + c], e)
    return y


def columns(n):
    """Columns in the first and the last sub-block of 16 and block of 64."""
    return sorted({0, 1, n // 2, n - 1} | {c for c in (17, 40, 70) if c < n})


@pytest.mark.parametrize("n", [5, 8, 12, 16, 20, 32, 33, 40, 65, 128])
@pytest.mark.parametrize("blocks", [(1, 3), (2,), (1, 2, 3, 4)])
@pytest.mark.parametrize("exponents", [(-1022,), (1022,), (-1022, 1022)])
def test_panels_with_single_extreme_pivots(n, blocks, exponents):
    """Pivots below 2^-1021 and from 2^1021 on: the LU kernels' reciprocal steps do
    not take them, so the panel is run again with correctly rounded reciprocals,
    from its first column or from that of a later sub-block or block.  cond(A) <=
    8e4 before the scaling (dense SVD) and entries rounded to 2^-52, that is 2e-11:
    bar 1e-9."""
    scales = {(k, c): exponents[i % len(exponents)] for k in blocks for i, c in enumerate(columns(n))}
    s, rhs, want = scaled_system(n, 5, scales, seed=n)
    for fused in (False, True):
        h = B.BorderedCR()
        h.load_system(s)
        h.select("LU")
        h.select_last("LU")
        x = rhs.copy()
        if fused:
            assert h.factorize_solve(2, x.reshape(-1), x.shape[1]), h.last_error()
        else:
            assert h.factorize(), h.last_error()
            assert h.solve_n(2, x.reshape(-1), x.shape[1]), h.last_error()
        assert fwd_err(unscale(s, x, scales)[:, :s.ncols], want[:, :s.ncols]) < 1e-9


@pytest.mark.parametrize("n", [5, 8, 12, 16, 20, 32])
@pytest.mark.parametrize("exponents", [(-126,), (126,), (-126, 126)])
def test_fp32_panels_with_single_extreme_pivots(n, exponents):
    """The same at the ends of the FP32 range.  The residual of such a system is
    measured against its largest entries, so the refinement stops with the FP32
    solution: cond(A) * 2^-23 <= 1.2e-4 (dense SVD), bar 1e-2."""
    scales = {(k, c): exponents[i % len(exponents)] for k in (1, 3) for i, c in enumerate(columns(n))}
    s, rhs, want = scaled_system(n, 5, scales, seed=n)
    h = B.BorderedCR()
    h.load_system(s)
    h.set_precision(B.PRECISION_MIXED)
    assert h.factorize(), h.last_error()
    x = rhs.copy()
    assert h.solve_n(2, x.reshape(-1), x.shape[1]), h.last_error()
    assert fwd_err(unscale(s, x, scales)[:, :s.ncols], want[:, :s.ncols]) < 1e-2


@pytest.mark.parametrize("n", [4, 16, 32, 33, 65, 128])
def test_last_block_with_extreme_pivots(n):
    """Unknowns of the first and the last block of the mesh scaled by 2^1021: their
    pivots are the last block's, of order 2n + 2.  Bar: as test_panels_with_single_extreme_pivots."""
    scales = {(k, c): 1021 for k in (0, 5) for c in columns(n)}
    s, rhs, want = scaled_system(n, 5, scales, seed=n)
    h = B.BorderedCR()
    h.load_system(s)
    h.select("LU")
    h.select_last("LU")
    assert h.factorize(), h.last_error()
    x = rhs.copy()
    assert h.solve_n(2, x.reshape(-1), x.shape[1]), h.last_error()
    assert fwd_err(unscale(s, x, scales)[:, :s.ncols], want[:, :s.ncols]) < 1e-9


@pytest.mark.parametrize("n", [1, 5, 12, 16])
@pytest.mark.parametrize("select", ["QR", "QRP"])
@pytest.mark.parametrize("panel,trail", [(-450, -600), (450, 600), (0, -1000), (0, 1000)])
def test_reflectors_on_columns_of_other_magnitudes(n, select, panel, trail):
    """Householder panels: one pair whose panel columns are scaled by 2^panel and
    whose other columns are scaled by 2^trail.  Products of elements of both leave
    the range, products with the scaled reflector do not.  cond(A) <= 1e3 (dense SVD)
    before the scaling: bar 1e-11, and the entries are scaled exactly."""
    scales = {(k, c): panel if k == 1 else trail for k in range(3) for c in range(n)}
    s, rhs, want = scaled_system(n, 2, scales, seed=n)
    h = B.BorderedCR()
    h.load_system(s)
    h.select(select)
    h.select_last("LU")
    assert h.factorize(), h.last_error()
    x = rhs.copy()
    assert h.solve_n(2, x.reshape(-1), x.shape[1]), h.last_error()
    assert fwd_err(unscale(s, x, scales)[:, :s.ncols], want[:, :s.ncols]) < 1e-11
