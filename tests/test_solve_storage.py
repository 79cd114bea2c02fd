"""Storage of the solves: a call for more right-hand sides than the device's memory holds is refused with
MFD_E_NOMEM, and the handle then solves as if it had not been made."""
import ctypes as C

import numpy as np
import pytest

from mfdag import hppllt as H
from mfdag import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", [0, 3])
@pytest.mark.parametrize("line", [24, 160])
@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("precision", [0, 1])
def test_solve_after_refused_allocation(precision, use_graph, line, before):
    """400 unknowns and 2^27 right-hand sides take 430 GB (FP32: 215 GB) for the solution alone.  `before`:
    right-hand sides of a solve before the refused one; `line` 24: with large fronts, 160: without."""
    p = P.laplace2d(20)
    s = H.Solver.analyze(p.n, p.col, p.row, p.order, max_zero=10, small_front_max=line, precision=precision,
                         use_graph=use_graph)
    assert s.factorize(p.val) == 0
    B = np.asfortranarray(np.random.default_rng(1).uniform(-1, 1, (p.n, 5)))

    def check(k):
        X = B[:, :k].copy(order="F")
        rep, rc = s.solve(X)
        assert rc == 0
        for r in range(k):
            assert P.backward_error(p.n, p.col, p.row, p.val, X[:, r], B[:, r]) <= 1e-12
        return X

    first = check(before) if before else None
    x = B[:, 0].copy()                                   # never read: the refusal comes first
    assert H.load().mfd_solve(s._h, x.ctypes.data, 1 << 27, p.n, None) == -3
    assert np.array_equal(x, B[:, 0])
    check(1)
    if before:
        assert np.array_equal(check(before), first)
    check(5)
    assert s.factorize(p.val) == 0
    check(1)
    s.close()
