"""GPU test of the accuracy of LU last blocks against LAPACK's."""
import numpy as np
import pytest

from alglin_b200 import bcr as B
from alglin_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,q,nr,seeds", [(16, 2, 4, 60), (64, 0, 16, 60), (128, 4, 16, 60)])
def test_last_block_is_as_accurate_as_lapack(n, q, nr, seeds):
    """One block, so that the last block is the whole matrix, of order 38 to 288: the
    errors of the solutions against the known one, relative to those of LAPACK's
    gesv.  One system's ratio has a standard deviation of about 0.5 (logarithm), the
    mean over 60 one of 0.065: the bar of 1.22 is three of them."""
    ratio = []
    h = B.BorderedCR()
    for seed in range(seeds):
        s = synth.collocation(1, n, q, q, nr, nr, seed=seed)
        A = s.to_dense()
        x = np.random.default_rng(1000 + seed).standard_normal(s.ncols)
        b = (A.astype(np.longdouble) @ x.astype(np.longdouble)).astype(np.float64)
        h.load_system(s)
        h.select_last("LU")
        assert h.factorize(), h.last_error()
        y = b.copy()
        assert h.solve(y), h.last_error()
        ratio.append(np.linalg.norm(y - x) / np.linalg.norm(np.linalg.solve(A, b) - x))
    assert np.exp(np.mean(np.log(ratio))) < 1.22
