"""GPU tests of a batch whose pair kernels are tuned between its factorization
and its solves, against the CPU oracle.

Bars: forward error <= 1e-10 in FP64, as in the other batch tests; the mixed path
is refined to a relative residual of 1e-15, which cond(A) <= 2e5 (dense SVD) turns
into 2e-10: forward error <= 1e-8."""
import numpy as np
import pytest

from alglin_b200 import bcr as B
from alglin_b200 import synth
from oracle import pyoracle as po
from tests._util import fwd_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", [B.BATCH_PERSISTENT, B.BATCH_LEVELS])
@pytest.mark.parametrize("precision", [B.PRECISION_FP64, B.PRECISION_MIXED])
@pytest.mark.parametrize("n", [4, 8, 16, 32])
def test_autotune_keeps_the_factorization(n, precision, schedule):
    """factorize -> autotune -> solve: the tuner tries several kernel families,
    which leave their factors in different forms; the solve has to take the form
    of the factors that are there.  Borders that the other tests do not tune, one
    pair per schedule, so that the tuner's choices of one case do not narrow the
    next one's."""
    nr = (3 if schedule == B.BATCH_PERSISTENT else 1) if precision == B.PRECISION_FP64 else \
        (4 if schedule == B.BATCH_PERSISTENT else 2)
    nx = 1 if nr == 3 else nr
    systems = [synth.collocation(nb, n, 0, nr - nx, nr, nx, seed=50 + i) for i, nb in enumerate((1, 9, 37, 20) if n == 32 else (1, 37, 90, 60))]
    rhs = [synth.rhs(s, 1, seed=70 + i)[0] for i, s in enumerate(systems)]
    hs = []
    for s in systems:
        h = B.BorderedCR()
        h.load_system(s)
        h.select("LU")
        h.select_last("LU")
        hs.append(h)
    want = []
    for s, b in zip(systems, rhs):
        o = po.Oracle(s, "LU", "LU")
        assert o.factorize(), o.last_error()
        want.append(o.solve(b[None, :])[0])
    mixed = precision == B.PRECISION_MIXED
    bt = B.Batch(hs)
    bt.set_schedule(schedule)
    bt.set_precision(precision)
    bt.set_refinement(1e-15, 30)
    bt.prepare()
    assert bt.factorize(), bt.last_error()
    for tune in (True, False):  # tuned after the factorization, then factorized with the choice
        if tune:
            bt.autotune()
        else:
            assert bt.factorize(), bt.last_error()
        xs = [b.copy() for b in rhs]
        assert bt.solve(xs), bt.last_error()
        if mixed:
            assert bt.refinement_info()[1] <= 1e-15
        for s, x, xo in zip(systems, xs, want):
            assert fwd_err(x[:s.ncols], xo[:s.ncols]) < (1e-8 if mixed else 1e-10)
