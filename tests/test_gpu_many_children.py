"""Large fronts with many children (bordered block-diagonal matrices): from kManyChildren = 32 on they add their
children from the children's side, in the factorization (k_add_children) and in the forward sweeps (k_gather_many),
below that from their own.  Counts at that line and at the edges of the 32 children that a warp looks at together,
children of 1 to 40 rows that overlap, fronts with and without rows below their columns."""
import numpy as np
import pytest

from mfdag import hppllt as H


def _bordered(leaves, mid, top, seed):
    """Leaf blocks of 1 to 4 columns coupled to up to 40 rows of the mid block and of the first half of the top
    block, which the mid block is coupled to as well.  Diagonally dominant; condition number below 10."""
    rng = np.random.default_rng(seed)
    sizes = rng.integers(1, 5, leaves)
    first = np.concatenate([[0], np.cumsum(sizes)])
    m0, t0 = int(first[-1]), int(first[-1]) + mid
    n = t0 + top
    a = np.zeros((n, n))
    for k in range(leaves):
        c = np.arange(first[k], first[k + 1])
        rows = np.concatenate([m0 + rng.choice(mid, rng.integers(1, min(mid, 30)), replace=False),
                               t0 + rng.choice(max(1, top // 2), rng.integers(0, min(top // 2, 10) + 1), replace=False)
                               if top else np.zeros(0, int)])
        a[np.ix_(c, c)] = rng.uniform(-1, 1, (c.size, c.size))
        a[np.ix_(rows, c)] = rng.uniform(-1, 1, (rows.size, c.size))
    a[m0:t0, m0:t0] = rng.uniform(-1, 1, (mid, mid))
    if top:
        a[t0:t0 + top // 2, m0:t0] = rng.uniform(-1, 1, (top // 2, mid))
        a[t0:, t0:] = rng.uniform(-1, 1, (top, top))
    a = np.tril(a, -1)
    a = a + a.T
    a[np.arange(n), np.arange(n)] = 1.25 * np.abs(a).sum(axis=1).max()
    low = np.tril(a)
    col, row = np.nonzero(low.T)
    ptr = np.concatenate([[1], 1 + np.cumsum(np.bincount(col, minlength=n))]).astype(np.int32)
    return a, ptr, (row + 1).astype(np.int32), low[row, col]


def _children(sym):
    p = np.asarray(sym["parent"])
    return np.bincount(p[p > 0] - 1, minlength=p.size)


@pytest.mark.parametrize("leaves", [31, 32, 33, 64, 65, 97])
@pytest.mark.parametrize("mid,top", [(170, 0), (161, 100), (300, 70)])
def test_structure(leaves, mid, top):
    """The mid block is a front of as many children as there are leaves, on either side of the line."""
    a, ptr, row, val = _bordered(leaves, mid, top, leaves)
    sym = H.symbolic_analyze(a.shape[0], ptr, row, np.arange(1, a.shape[0] + 1, dtype=np.int32), 0)
    k = int(np.argmax(_children(sym)))
    assert _children(sym)[k] == leaves
    nc, nr = np.diff(sym["node_ptr"])[k], np.diff(sym["lptr"])[k]
    assert nc >= 128 and nc + nr > 160 and (nr > 0) == (top > 0)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("leaves", [31, 32, 33, 64, 65, 97])
@pytest.mark.parametrize("mid,top", [(170, 0), (161, 100), (300, 70)])
def test_many_children_against_dense(mid, top, leaves, precision):
    """Against numpy's dense solve with 1, 3, 8, 9 and 17 right-hand sides: both in FP64 and backward stable at a
    condition number below 10, 1e-12; FP32 + refinement to a backward error of 1e-12, 1e-10.  The sweeps of one
    launch per panel step gather on their own and give the same within that."""
    a, ptr, row, val = _bordered(leaves, mid, top, leaves)
    n = a.shape[0]
    order = np.arange(1, n + 1, dtype=np.int32)
    tol = 1e-12 if precision == 0 else 1e-10
    B = np.asfortranarray(np.random.default_rng(7).uniform(-1, 1, (n, 17)))
    want = np.linalg.solve(a, B)
    for per_step in (0, 1):
        s = H.Solver.analyze(n, ptr, row, order, max_zero=0, precision=precision, reserved=(0, 0, 0, 0, 0, 0, per_step))
        assert s.factorize(val) == 0
        for k in (1, 3, 8, 9, 17):
            X = B[:, :k].copy(order="F")
            rep, rc = s.solve(X)
            assert rc == 0
            assert np.abs(X - want[:, :k]).max() <= tol * np.abs(want).max(), k
        s.close()
