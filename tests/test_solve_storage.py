"""Calls that the device has no memory for are refused with MFD_E_NOMEM, and the handle then works as if they had
not been made; what is only there for speed is done without.  Storage of the solves: more right-hand sides than the
device holds.  Every single allocation of the set-up and of a first solve: refused by request."""
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


def _dense(n):
    """Eigenvalues within [n / 2, 3 n / 2] or so; one front."""
    a = np.random.default_rng(n).uniform(-1.0, 1.0, (n, n))
    a = (a + a.T) * (np.sqrt(n) / 8.0) + n * np.eye(n)
    col = np.concatenate([[1], 1 + np.cumsum(np.arange(n, 0, -1))]).astype(np.int32)
    row = np.concatenate([np.arange(j + 1, n + 1) for j in range(n)]).astype(np.int32)
    return col, row, np.concatenate([a[j:, j] for j in range(n)])


def _problems():
    p = P.laplace2d(20)
    col, row, val = _dense(1153)                         # its first update step reads packed operands, in FP64 too
    return {"laplace": (p.n, p.col, p.row, p.order, p.val, dict(max_zero=10, small_front_max=24)),
            "dense": (1153, col, row, None, val, dict(max_zero=0))}


@pytest.mark.parametrize("which,precision", [("laplace", 0), ("laplace", 1), ("dense", 0), ("dense", 1)])
def test_every_allocation_refused_once(which, precision):
    """In the set-up only the packed update operands can be done without: FP64 solutions then keep their bits, FP32 +
    refinement its backward error.  In a first solve everything is needed, but those operands are given up for it;
    the handle solves, factors and solves after either outcome."""
    n, col, row, order, val, opts = _problems()[which]
    opts["precision"] = precision
    L = H.load()
    b = np.random.default_rng(3).uniform(-1, 1, n)

    def solve(s):
        x = b.copy()
        rep, rc = s.solve(x)
        assert rc == 0 and P.backward_error(n, col, row, val, x, b) <= (1e-14 if precision == 0 else 1e-12)
        return x

    def same(x, y):
        assert np.array_equal(x, y) if precision == 0 else np.abs(x - y).max() <= 1e-9 * np.abs(y).max()

    try:
        L.mfd_test_fail_alloc(0)
        s = H.Solver.analyze(n, col, row, order, **opts)
        in_setup = L.mfd_test_fail_alloc(0)
        assert s.factorize(val) == 0 and L.mfd_test_fail_alloc(0) == 0
        ref = solve(s)
        in_solve = L.mfd_test_fail_alloc(0)
        s.close()
        assert in_setup > 20 and in_solve >= 1
        without = 0
        for k in range(1, in_setup + 1):
            L.mfd_test_fail_alloc(k)
            try:
                s = H.Solver.analyze(n, col, row, order, **opts)
            except H.MfdError as e:
                assert e.code == -3
                continue
            finally:
                L.mfd_test_fail_alloc(0)
            without += 1
            assert s.factorize(val) == 0
            same(solve(s), ref)
            s.close()
        packed = which == "dense" or precision == 1
        assert without == (1 if packed else 0)
        for k in range(1, in_solve + 1):
            s = H.Solver.analyze(n, col, row, order, **opts)
            assert s.factorize(val) == 0
            L.mfd_test_fail_alloc(k)
            x = b.copy()
            rc = L.mfd_solve(s._h, x.ctypes.data, 1, n, None)
            L.mfd_test_fail_alloc(0)
            assert rc == (0 if packed else -3), k
            same(solve(s), ref)
            assert s.factorize(val) == 0
            same(solve(s), ref)
            s.close()
    finally:
        L.mfd_test_fail_alloc(0)
