"""Blocked large-front kernels at the sizes where their tiling can go wrong.

* Panel step (POTRF on 8 x 8 blocks, block-substitution TRSM): dense fronts
  whose column counts sit at the edges of 8, 32 and 128, with and without rows
  below, against numpy.  A backward-stable factorization of a matrix with
  condition number below 10 differs from another by a modest multiple of
  n eps: 1e-12 relative is 8 n eps at the largest n here.
* Several-right-hand-side sweeps (tiles of eight): counts at the tile's edges
  against the per-step sweeps on the same factor.
"""
import numpy as np
import pytest

from helpers import lower_panel
from mfdag import hppllt as H
from mfdag import problems as P

pytestmark = pytest.mark.gpu


def _spd(n, seed):
    """Symmetric, eigenvalues within [n / 2, 3 n / 2] or so."""
    a = np.random.default_rng(seed).uniform(-1.0, 1.0, (n, n))
    return (a + a.T) * (np.sqrt(n) / 8.0) + n * np.eye(n)


@pytest.mark.parametrize("nf,nc", [(1, 1), (7, 7), (8, 8), (9, 9), (31, 31), (33, 33), (65, 64), (97, 96), (127, 127),
                                   (128, 128), (129, 129), (130, 1), (136, 128), (137, 9), (200, 63), (257, 128),
                                   (300, 129), (333, 250), (400, 136)])
def test_dense_partial_factor(nf, nc):
    import torch
    a = _spd(nf, nf * 1000 + nc)
    nr = nf - nc
    panel = np.asfortranarray(np.tril(a)[:, :nc])
    upd = np.asfortranarray(np.tril(a[nc:, nc:]))
    off = (nf * nc + 31) // 32 * 32
    buf = np.zeros(off + max(1, nr * nr))
    buf[:nf * nc] = panel.ravel(order="F")
    buf[off:off + nr * nr] = upd.ravel(order="F")
    d = torch.from_numpy(buf).cuda()
    assert H.factor_fronts_noalloc(d, [0], [off], [nf], [nc]) == 0
    got = d.cpu().numpy()
    L = np.linalg.cholesky(a[:nc, :nc])
    X = np.linalg.solve(L, a[nc:, :nc].T).T
    want = np.vstack([L, X])
    P_ = np.tril(got[:nf * nc].reshape((nf, nc), order="F"))
    assert np.abs(P_ - np.tril(want)).max() <= 1e-12 * np.abs(want).max()
    if nr:
        U = np.tril(got[off:off + nr * nr].reshape((nr, nr), order="F"))
        S = np.tril(a[nc:, nc:] - X @ X.T)
        assert np.abs(U - S).max() <= 1e-12 * np.abs(S).max()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nrhs", [2, 7, 8, 9, 33])
def test_several_rhs_sweeps_match_per_step(nrhs, precision):
    """3D Laplacian 20^3 with fronts above 48 rows on the blocked path (panel
    steps of full and partial width, update-row chunks of full and partial
    height).  FP64: both sweeps are backward stable and the condition number is
    below 300, so they agree within 1e-12; FP32 + refinement: backward error
    1e-12 each.  A second solve gives the same bits."""
    p = P.laplace3d(20)
    B = np.asfortranarray(np.random.default_rng(nrhs).uniform(-1, 1, (p.n, nrhs)))
    xs = []
    for per_step in (0, 1):
        s = H.Solver.analyze(p.n, p.col, p.row, p.order, max_zero=1000, small_front_max=48, precision=precision,
                             reserved=(0, 0, 0, 0, 0, 0, per_step))
        assert s.factorize(p.val) == 0
        X = B.copy(order="F")
        rep, rc = s.solve(X)
        assert rc == 0
        for r in range(nrhs):
            assert P.backward_error(p.n, p.col, p.row, p.val, X[:, r], B[:, r]) <= (1e-14 if precision == 0 else 1e-12)
        if per_step == 0:
            Y = B.copy(order="F")
            s.solve(Y)
            assert np.array_equal(X, Y)
            x1 = B[:, 0].copy()                          # fewer right-hand sides on the same handle afterwards
            s.solve(x1)
            assert P.backward_error(p.n, p.col, p.row, p.val, x1, B[:, 0]) <= 1e-12
        xs.append(X)
        s.close()
    assert np.abs(xs[0] - xs[1]).max() <= (1e-12 if precision == 0 else 1e-9) * np.abs(xs[1]).max()


@pytest.mark.parametrize("precision", [0, 1])
def test_several_rhs_expired_wait(precision):
    """A sweep's flag wait that runs out ends the solve with MFD_E_TIMEOUT; the handle solves afterwards."""
    p = P.laplace3d(16)
    s = H.Solver.analyze(p.n, p.col, p.row, p.order, max_zero=1000, small_front_max=48, precision=precision)
    assert s.factorize(p.val) == 0
    B = np.asfortranarray(np.random.default_rng(0).uniform(-1, 1, (p.n, 10)))
    s.test_expire_waits(True)
    with pytest.raises(H.MfdError) as e:
        s.solve(B.copy(order="F"))
    assert e.value.code == -4
    s.test_expire_waits(False)
    X = B.copy(order="F")
    rep, rc = s.solve(X)
    assert rc == 0
    assert P.backward_error(p.n, p.col, p.row, p.val, X[:, 9], B[:, 9]) <= 1e-12


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 5, 15, 16, 17, 24, 25, 32, 33, 57, 64, 65, 89, 96, 97, 128, 129, 153, 160, 161])
def test_small_front_sizes(n, precision):
    """One dense front of n rows and columns: the edges of the one-warp sizes
    (16, 24, 32), of the one-CTA sizes (64, 96, 128, 160), of their 8-column
    blocks, and the first size of the blocked path.  Backward error against the
    dense product: FP64 n eps, FP32 + refinement 1e-12."""
    a = _spd(n, n)
    col, rows, vals = [1], [], []
    for j in range(n):
        rows.extend(range(j + 1, n + 1))
        vals.extend(a[j:, j])
        col.append(len(rows) + 1)
    s = H.Solver.analyze(n, np.array(col), np.array(rows), None, max_zero=0, precision=precision)
    assert s.stats().num_front == 1
    assert s.factorize(np.array(vals)) == 0
    B = np.asfortranarray(np.random.default_rng(n).uniform(-1, 1, (n, 3)))
    for X in (B[:, 0].copy(), B.copy(order="F")):
        b = X.copy(order="F")
        rep, rc = s.solve(X)
        assert rc == 0
        r = np.abs(b - a @ X).max()
        den = np.abs(a).sum(axis=1).max() * np.abs(X).max() + np.abs(b).max()
        assert r / den <= (1e-14 if precision == 0 else 1e-12)


@pytest.mark.parametrize("n", [1153, 2049, 2190])
def test_packed_fp64_update_bitwise(n):
    """A dense front long enough for the packed-operand FP64 update (its trailing
    triangle in 128 x 64 pieces reaches half of the SMs; 1153 rows: 90 pieces in the
    first step, the last row block with one row, and too few from the second on),
    full and partial last panel: the
    factor is bit for bit the one of the whole-tile kernel that reads the panel
    (reserved[0] = 3), with the lookahead on and off, and with either deferral
    depth; its backward error is at most 1e-14."""
    a = _spd(n, n)
    col = np.concatenate([[1], 1 + np.cumsum(np.arange(n, 0, -1))]).astype(np.int32)
    rows = np.concatenate([np.arange(j + 1, n + 1) for j in range(n)]).astype(np.int32)
    vals = np.concatenate([a[j:, j] for j in range(n)])
    b = np.random.default_rng(1).uniform(-1, 1, n)
    panels = {}
    for kind, lookahead_off, defer in ((0, 0, 2), (0, 1, 2), (3, 0, 2), (0, 0, 1)):
        s = H.Solver.analyze(n, col, rows, None, max_zero=0, reserved=(kind, lookahead_off, 0, 0, 0, defer, 0))
        assert s.factorize(vals) == 0
        x = b.copy()
        s.solve(x)
        den = np.abs(a).sum(axis=1).max() * np.abs(x).max() + np.abs(b).max()
        assert np.abs(b - a @ x).max() / den <= 1e-14
        panels[kind, lookahead_off, defer] = np.tril(s.front_panel(1).reshape((n, n), order="F"))
        s.close()
    ref = panels.pop((3, 0, 2))
    for key, p in panels.items():
        assert np.array_equal(p, ref), key


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("n,lookahead_off", [(1153, 1), (2049, 0)])
def test_packed_fp64_update_expired_wait(n, lookahead_off, use_graph):
    """The packed-operand FP64 update's bounded wait runs out with its copies in flight (the request makes it wait
    on a barrier of its own): the factorization ends with MFD_E_TIMEOUT, there is no factor to solve with, and the
    handle factors as before, bit for bit, once the request is withdrawn.  1153 rows: 90 pieces in the first step as
    one launch, too few for packed operands where the lookahead splits it; 2049 rows: 240 in its second part.  Not
    packed (reserved[0] = 3): no wait."""
    a = _spd(n, n)
    col = np.concatenate([[1], 1 + np.cumsum(np.arange(n, 0, -1))]).astype(np.int32)
    rows = np.concatenate([np.arange(j + 1, n + 1) for j in range(n)]).astype(np.int32)
    vals = np.concatenate([a[j:, j] for j in range(n)])
    s = H.Solver.analyze(n, col, rows, None, max_zero=0, use_graph=use_graph, reserved=(0, lookahead_off, 0, 0, 0, 0, 0))
    assert s.factorize(vals) == 0
    ref = s.front_panel(1).copy()
    for _ in range(2):
        s.test_expire_waits(True)
        with pytest.raises(H.MfdError) as e:
            s.factorize(vals)
        assert e.value.code == -4
        with pytest.raises(H.MfdError) as e:
            s.solve(np.ones(n))
        assert e.value.code == -6
        s.test_expire_waits(False)
        assert s.factorize(vals) == 0
        assert np.array_equal(s.front_panel(1), ref)
    s.close()
    s = H.Solver.analyze(n, col, rows, None, max_zero=0, use_graph=use_graph, reserved=(3, 0, 0, 0, 0, 0, 0))
    s.test_expire_waits(True)
    assert s.factorize(vals) == 0
    s.close()


def _dense_ccs(n):
    a = _spd(n, n)
    col = np.concatenate([[1], 1 + np.cumsum(np.arange(n, 0, -1))]).astype(np.int32)
    rows = np.concatenate([np.arange(j + 1, n + 1) for j in range(n)]).astype(np.int32)
    return a, col, rows, np.concatenate([a[j:, j] for j in range(n)])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sizes", [(161, 384, 641, 1153), (1537, 1500, 129 * 9, 512, 385, 200), (2049, 1025, 1024, 1023)])
def test_packed_updates_of_fronts_that_end_at_different_steps(sizes, precision):
    """Dense systems of different orders in one handle: one level of fronts that leave the panel steps one after
    another, so that a step's packed rows hold fewer fronts than the one's before and the deferred groups end at
    different steps.  FP64: bit for bit the factor of the whole-tile kernel that reads the panel; FP32 + refinement:
    a backward error of 1e-12, with the number of sweeps of the unpacked form (deferral 4) or one more."""
    parts = [_dense_ccs(n) for n in sizes]
    systems = [(n, p[1], p[2], None) for n, p in zip(sizes, parts)]
    vals = np.concatenate([p[3] for p in parts])
    b = np.random.default_rng(2).uniform(-1, 1, sum(sizes))
    schedules = [(0, 0, 0), (0, 1, 0), (0, 0, 1), (0, 0, 2), (0, 1, 2), (3, 0, 0)] if precision == 0 else [(0, 0, 1), (0, 0, 2), (0, 1, 2), (0, 0, 4)]
    got = {}
    for kind, lookahead_off, defer in schedules:
        s = H.Solver.analyze_batch(systems, max_zero=0, precision=precision,
                                   reserved=(kind, lookahead_off, 0, 0, 0, defer, 0))
        for _ in range(2):                               # launched, then as a graph
            assert s.factorize(vals) == 0
        x = b.copy()
        rep, rc = s.solve(x)
        assert rc == 0
        at = 0
        for n, p in zip(sizes, parts):
            xs, bs = x[at:at + n], b[at:at + n]
            den = np.abs(p[0]).sum(axis=1).max() * np.abs(xs).max() + np.abs(bs).max()
            assert np.abs(bs - p[0] @ xs).max() / den <= (1e-14 if precision == 0 else 1e-12)
            at += n
        panels = [np.tril(s.front_panel(1, system=k).reshape((n, n), order="F")) for k, n in enumerate(sizes)]
        got[kind, lookahead_off, defer] = (panels, rep.iterations)
        s.close()
    if precision == 0:
        for key, (panels, _) in got.items():
            for p, q in zip(panels, got[3, 0, 0][0]):
                assert np.array_equal(p, q), key
    else:
        for key, (_, sweeps) in got.items():
            assert sweeps <= got[0, 0, 4][1] + 1, key


def test_packed_fp64_update_in_a_tree():
    """A 3D Laplacian whose upper levels pack their operands (fronts of up to 1,296 columns, with update rows, several
    to a level) and whose lower ones do not: the same bits as with the whole-tile kernel that reads the panel."""
    p = P.laplace3d(36)
    sym = H.symbolic_analyze(p.n, p.col, p.row, p.order, 1000)
    nc, nr = np.diff(sym["node_ptr"]), np.diff(sym["lptr"])
    b = np.random.default_rng(4).uniform(-1, 1, p.n)
    got = []
    for kind, lookahead_off, defer in ((3, 0, 0), (0, 0, 0), (0, 1, 2), (0, 0, 1)):
        s = H.Solver.analyze(p.n, p.col, p.row, p.order, max_zero=1000, reserved=(kind, lookahead_off, 0, 0, 0, defer, 0))
        assert s.factorize(p.val) == 0
        x = b.copy()
        s.solve(x)
        assert s.stats().num_front == nc.size
        got.append([x] + [lower_panel(s.front_panel(f + 1), int(nc[f] + nr[f]), int(nc[f])) for f in range(nc.size - 40, nc.size)])
        s.close()
    for other in got[1:]:
        for u, v in zip(got[0], other):
            assert np.array_equal(u, v)
