"""GPU parity tests: the sm_100a path through the C ABI against the CPU oracle.

Integer index data (local_index, supernodal_index, block_local_index) must be
bit-exact; FP64 factors and solutions within the tolerances written below;
FP32 + FP64 iterative refinement to backward error <= 1e-12.
"""
import json
import os

import numpy as np
import pytest

from golden import reference_vectors as R
from helpers import lower_panel, oracle_front_panel, toy_symbolic
from mfdag import hppllt as H
from mfdag import problems as P
from oracle import oracle as O

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))

FP64_X_TOL = 1e-10        # ||x - x_oracle||_inf / ||x_oracle||_inf (both FP64, different summation order)
FP64_BWD_TOL = 1e-12      # normwise backward error target
FACTOR_TOL = 1e-12        # relative entrywise difference of factor panels


def oracle_for(p, nb=10, max_zero=10):
    o = O.Oracle.analyze(p.n, p.col, p.row, nb=nb, max_zero=max_zero, order_perm=p.order)
    assert o.factorize(p.val) == 0
    return o


def gpu_for(p, max_zero=10, **opts):
    s = H.Solver.analyze(p.n, p.col, p.row, p.order, max_zero=max_zero, **opts)
    assert s.factorize(p.val) == 0
    return s


# ---------------------------------------------------------------------------
# the reference's own numeric fixture
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("nb", [2, 3])
def test_toy_factor_matches_reference_vectors(nb):
    sym = toy_symbolic()
    s = H.Solver.from_symbolic(sym, nb=nb)
    assert s.factorize(np.array(R.TOY_VALUES, np.float64)) == 0
    o = O.Oracle.from_internal(R.TOY_NODE_SIZE, [len(x) for x in sym["lrows"]], sym["lrow"], R.TOY_PARENT, 13,
                               sym["aptr"], sym["arow"], nb)
    assert o.factorize(np.array(R.TOY_VALUES, np.float64)) == 0
    for node in (1, 2, 3):
        nc, nr = R.TOY_NODE_SIZE[node - 1], R.TOY_WORK_SIZE[node - 1]
        got = lower_panel(s.front_panel(node), nc + nr, nc)
        ref = oracle_front_panel(o, node, nc, nr, nb)
        assert np.allclose(got, ref, rtol=0, atol=1e-12), node
        assert np.array_equal(np.round(got), ref)          # the fixture's factor is integer-valued
    # index data built on the device
    assert list(s.index(H.LOCAL_INDEX)) == R.TOY_LOCAL_VAL
    assert list(s.index(H.SUPERNODAL_INDEX)) == R.TOY_SIDX_VAL


@pytest.mark.parametrize("nb", [2, 3])
def test_toy_solve(nb):
    sym = toy_symbolic()
    s = H.Solver.from_symbolic(sym, nb=nb)
    assert s.factorize(np.array(R.TOY_VALUES, np.float64)) == 0
    # A x = b with x = 1: b = L L^T 1 from the oracle's sweeps run backwards is not
    # available, so build A from the values and check the residual directly
    n = 13
    A = np.zeros((n, n))
    for j in range(n):
        for k in range(sym["aptr"][j] - 1, sym["aptr"][j + 1] - 1):
            r = sym["arow"][k] - 1
            A[r, j] = A[j, r] = R.TOY_VALUES[k]
    x_true = np.arange(1, n + 1, dtype=np.float64)
    b = A @ x_true
    x = b.copy()
    rep, rc = s.solve(x)
    assert rc == 0
    assert np.allclose(x, x_true, rtol=1e-12, atol=1e-12)


# ---------------------------------------------------------------------------
# index maps: bit-exact with the oracle (reference semantics)
# ---------------------------------------------------------------------------
def index_cases():
    yield "lap2d_30", P.laplace2d(30), 10, 10
    yield "lap2d_30_nb4", P.laplace2d(30), 4, 10
    yield "lap3d_12", P.laplace3d(12), 10, 10
    yield "lap3d_12_mz1000", P.laplace3d(12), 7, 1000
    yield "diff3d_10", P.diffusion3d(10), 10, 10


@pytest.mark.parametrize("name,p,nb,mz", list(index_cases()), ids=[c[0] for c in index_cases()])
def test_index_maps_bit_exact(name, p, nb, mz):
    s = H.Solver.analyze(p.n, p.col, p.row, p.order, max_zero=mz, nb=nb)
    o = O.Oracle.analyze(p.n, p.col, p.row, nb=nb, max_zero=mz, order_perm=p.order)
    assert np.array_equal(s.index(H.LOCAL_INDEX), o.get(O.LOCAL))
    assert np.array_equal(s.index(H.SUPERNODAL_INDEX), o.get(O.SIDX))
    assert np.array_equal(s.index(H.BLI_NODE_PTR), o.get(O.BLI_NODE_PTR))
    assert np.array_equal(s.index(H.BLI_BLOCK_PTR), o.get(O.BLI_BLOCK_PTR))
    assert np.array_equal(s.index(H.BLI_PARENT), o.get(O.BLI_PARENT))
    assert np.array_equal(s.index(H.BLI_CHILD), o.get(O.BLI_CHILD))
    assert np.array_equal(s.index(H.BLI_VAL), o.get(O.BLI_VAL))
    assert np.array_equal(s.index(H.BLI_OFFSET), o.get(O.BLI_OFFSET))


# ---------------------------------------------------------------------------
# FP64 factor + solve
# ---------------------------------------------------------------------------
def check_solution(p, s, o, tol=FP64_X_TOL):
    x = p.rhs.copy()
    rep, rc = s.solve(x)
    assert rc == 0
    xo = o.solve(p.rhs)
    rel = np.abs(x - xo).max() / np.abs(xo).max()
    assert rel <= tol, rel
    bwd = P.backward_error(p.n, p.col, p.row, p.val, x, p.rhs)
    assert bwd <= FP64_BWD_TOL, bwd
    assert rep.backward_error <= FP64_BWD_TOL
    # the device residual and the host residual round differently at the 1e-16 level
    assert abs(rep.backward_error - bwd) <= 0.5 * max(bwd, rep.backward_error) + 1e-17
    return x


def test_laplace2d_100_fp64():                 # 2D 5-point, 100x100 (n = 10,000), x* from seed 0
    p = P.laplace2d(100)
    check_solution(p, gpu_for(p), oracle_for(p))


@pytest.mark.parametrize("small_max", [0, 48])
def test_laplace3d_fp64_large_path(small_max):
    """16^3 Laplacian; small_front_max=48 forces the blocked large-front kernels
    (zero/assemble/extend-add/panel/update) onto many fronts."""
    p = P.laplace3d(16)
    s = gpu_for(p, max_zero=10, small_front_max=small_max)
    o = oracle_for(p)
    check_solution(p, s, o)
    # factor panels of the largest fronts against the oracle's tiles
    sym = o.symbolic()
    nc = np.diff(sym["node_ptr"]); nr = np.diff(sym["lptr"])
    for node in np.argsort(-(nc + nr))[:3] + 1:
        a, b = int(nc[node - 1]), int(nr[node - 1])
        got = lower_panel(s.front_panel(int(node)), a + b, a)
        ref = oracle_front_panel(o, int(node), a, b, 10)
        assert np.abs(got - ref).max() <= FACTOR_TOL * np.abs(ref).max()


@pytest.mark.parametrize("precision", [0, 1])
def test_wide_panels_many_rows(precision):
    """22^3 Laplacian with large relaxed supernodes (max_zero 1000): fronts with
    several full 128-column panel steps and hundreds of rows below them, the
    shape where a panel step's POTRF, TRSM and trailing-update CTAs work on
    the same columns."""
    p = P.laplace3d(22)
    s = gpu_for(p, max_zero=1000, precision=precision)
    assert s.stats().max_front > 3 * 128
    x = p.rhs.copy()
    rep, rc = s.solve(x)
    assert rc == 0
    bwd = P.backward_error(p.n, p.col, p.row, p.val, x, p.rhs)
    assert bwd <= FP64_BWD_TOL, bwd
    if precision == 1:
        assert rep.iterations <= 3, rep.iterations
    xo = oracle_for(p, max_zero=1000).solve(p.rhs)
    assert np.abs(x - xo).max() <= 1e-9 * np.abs(xo).max()


def test_update_kernel_variants_agree():
    """FP64 trailing-update variants: the 128 x 64 half-tile DMMA kernel (the
    default) and the whole-tile one apply the same DMMA sequence to every
    entry (bit-identical); the FFMA tiles agree to rounding."""
    p = P.laplace3d(14)
    s0 = gpu_for(p, small_front_max=40)
    s1 = gpu_for(p, small_front_max=40, reserved=(1, 0, 0, 0, 0, 0, 0))
    s3 = gpu_for(p, small_front_max=40, reserved=(3, 0, 0, 0, 0, 0, 0))
    x0, x1, x3 = p.rhs.copy(), p.rhs.copy(), p.rhs.copy()
    s0.solve(x0)
    s1.solve(x1)
    s3.solve(x3)
    assert np.array_equal(x0, x3)
    assert np.abs(x0 - x1).max() <= 1e-12 * np.abs(x0).max()


def test_dense_front_update_variants_bitwise():
    """One dense front (n = 700: six panel steps, tiles on both sides of the
    panel / update-matrix boundary with a partial last panel, max_zero = 0)
    factored with both DMMA update kernels: identical factors; the solution
    matches numpy's."""
    n = 700
    rng = np.random.default_rng(12)
    M = rng.standard_normal((n, n))
    A = M @ M.T / n + 2.0 * np.eye(n)
    col, row, val = _dense_lower_ccs(A)
    out = []
    for kind in (0, 3):
        s = H.Solver.analyze(n, col, row, None, max_zero=0, reserved=(kind, 0, 0, 0, 0, 2, 0))
        assert s.factorize(val) == 0
        out.append(s.front_panel(1))
        b = A @ np.ones(n)
        x = b.copy()
        rep, rc = s.solve(x)
        assert rc == 0 and np.abs(x - 1.0).max() <= 1e-10
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("precision", [0, 1])
def test_lookahead_bitwise_equal(precision):
    """The lookahead schedule (next panel's update tiles on the main stream,
    the rest on a side stream) applies the same tile updates in the same order
    per entry as the serial schedule: identical factors and solutions."""
    p = P.laplace3d(16)
    s0 = gpu_for(p, precision=precision, small_front_max=48)
    s1 = gpu_for(p, precision=precision, small_front_max=48, reserved=(0, 1, 0, 0, 0, 0, 0))
    x0, x1 = p.rhs.copy(), p.rhs.copy()
    s0.solve(x0)
    s1.solve(x1)
    assert np.array_equal(x0, x1)


@pytest.mark.parametrize("precision", [0, 1])
def test_deferred_updates_bitwise_equal(precision):
    """Deferred trailing updates (reserved[5] = D: the bulk of the trailing
    matrix takes D panel steps' updates in one pass, the next panel catches up
    every step) apply every panel step to every entry once and in step order.
    For each D the lookahead schedule and the serial one give bit-identical
    solutions (fronts of 2, 4 and 9 panel steps, partial last panels).  In
    FP64 the accumulators start from C, so D = 1..4 are bit-identical too; the
    FP32 tensor-core update accumulates each pass from zero in TMEM and
    subtracts at the end, so there D changes the rounding and the refined
    solutions agree to the refinement tolerance.  All match the oracle."""
    p = P.laplace3d(32)
    outs = {}
    for d in (1, 2, 3, 4):
        for la in (0, 1):
            s = gpu_for(p, max_zero=1000, precision=precision, reserved=(0, la, 0, 0, 0, d, 0))
            x = p.rhs.copy()
            rep, rc = s.solve(x)
            assert rc == 0
            outs[d, la] = x
            s.close()
        assert np.array_equal(outs[d, 0], outs[d, 1]), d
    x1 = outs[1, 0]
    for d in (2, 3, 4):
        if precision == 0:
            assert np.array_equal(x1, outs[d, 0]), d
        else:
            assert np.abs(outs[d, 0] - x1).max() <= 1e-9 * np.abs(x1).max(), d
    xo = oracle_for(p, max_zero=1000).solve(p.rhs)
    assert np.abs(x1 - xo).max() <= (FP64_X_TOL if precision == 0 else 1e-8) * np.abs(xo).max()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("mk", [lambda: P.laplace3d(24), lambda: P.diffusion3d(16)], ids=["lap3d24", "diff3d16"])
def test_fused_solve_sweeps_match_per_step(mk, precision):
    """The single-RHS large-front sweeps run as one launch per level (tasks in
    dependency order, device flags; the update rows of the backward sweep in
    256-row chunk tasks) and, with reserved[6] = 1, one launch per panel step.
    Both give the oracle's solution (FP64: within the FP64 tolerance; FP32 +
    refinement: backward error <= 1e-12), agree with each other, and the fused
    form is deterministic (a second solve is bit-identical)."""
    p = mk()
    o = oracle_for(p, max_zero=1000)
    xs = {}
    for per_step in (0, 1):
        s = gpu_for(p, max_zero=1000, small_front_max=48, precision=precision,
                    reserved=(0, 0, 0, 0, 0, 0, per_step))
        x = p.rhs.copy()
        rep, rc = s.solve(x)
        assert rc == 0 and rep.backward_error <= FP64_BWD_TOL
        assert P.backward_error(p.n, p.col, p.row, p.val, x, p.rhs) <= FP64_BWD_TOL
        if per_step == 0:
            x2 = p.rhs.copy()
            s.solve(x2)
            assert np.array_equal(x, x2)
        xs[per_step] = x
        s.close()
    xo = o.solve(p.rhs)
    scale = np.abs(xo).max()
    for x in xs.values():
        # FP32 + refinement stops at backward error 1e-12: its forward error scales with the conditioning
        assert np.abs(x - xo).max() / scale <= (FP64_X_TOL if precision == 0 else 1e-6)
    assert np.abs(xs[0] - xs[1]).max() / scale <= (FP64_X_TOL if precision == 0 else 1e-6)


def test_programmatic_launch_matches():
    """Programmatic dependent launch along the panel chain (opt-in) gives the
    same factor as the default schedule."""
    p = P.laplace3d(22)
    s0 = gpu_for(p, max_zero=1000)
    s1 = gpu_for(p, max_zero=1000, reserved=(0, 0, 1, 0, 0, 0, 0))
    x0, x1 = p.rhs.copy(), p.rhs.copy()
    s0.solve(x0)
    s1.solve(x1)
    assert np.array_equal(x0, x1)


@pytest.mark.parametrize("precision", [0, 1])
def test_side_stream_levels_bitwise_equal(precision):
    """A level's small-front size bins on side streams next to its large
    fronts (the default) and the same launches on one stream (reserved[4] = 1)
    touch disjoint data: identical factors and solutions, single and several
    right-hand sides, on a batch with all four size bins in most levels."""
    systems = P.laplace2d_batch(12, 5)
    outs = []
    for res in ((0, 0, 0, 0, 0, 0, 0), (0, 0, 0, 0, 1, 0, 0)):
        s = H.Solver.analyze_batch([(q.n, q.col, q.row, q.order) for q in systems], max_zero=100,
                                   precision=precision, reserved=res)
        vals = np.concatenate([q.val for q in systems])
        assert s.factorize(vals) == 0
        b = np.concatenate([q.rhs for q in systems])
        x1 = b.copy()
        s.solve(x1)
        xm = np.asfortranarray(b[:, None] * np.arange(1, 10)[None, :])
        s.solve(xm, nrhs=9)
        outs.append((x1, xm))
        s.close()
    assert np.array_equal(outs[0][0], outs[1][0])
    assert np.array_equal(outs[0][1], outs[1][1])


def test_autotune_picks_a_candidate():
    """The autotuner times the schedule candidates and returns options whose
    handle factors to the same solution quality."""
    p = P.laplace3d(16)
    s = gpu_for(p, max_zero=1000)
    opts, ms = s.autotune(p.val, repeats=1)
    assert opts["small_front_max"] in (32, 64, 96, 128, 160) and ms > 0
    assert opts["reserved"][0] in (0, 1, 3) and opts["reserved"][5] in (0, 1, 2)
    t = gpu_for(p, max_zero=1000, **opts)
    x = p.rhs.copy()
    rep, rc = t.solve(x)
    assert rc == 0 and P.backward_error(p.n, p.col, p.row, p.val, x, p.rhs) <= FP64_BWD_TOL


@pytest.mark.parametrize("precision", [0, 1])
def test_autotune_times_the_default(precision):
    """The default schedule is one of the candidates: what the autotuner reports as the fastest is not slower than
    an untuned handle beyond the 3 % that a candidate has to gain and the noise of a factorization of about a
    millisecond (15 %; medians of nine)."""
    p = P.laplace3d(24)
    s = gpu_for(p, max_zero=1000, precision=precision)
    opts, ms = s.autotune(p.val, repeats=9)
    f = []
    for _ in range(11):
        assert s.factorize(p.val) == 0
        f.append(s.stats().factor_ms)
    assert ms <= 1.15 * np.median(f[2:])


def test_multiple_rhs():
    p = P.laplace2d(40)
    s = gpu_for(p)
    o = oracle_for(p)
    rng = np.random.default_rng(7)
    B = np.asfortranarray(rng.uniform(-1, 1, (p.n, 3)))
    X = B.copy(order="F")
    rep, rc = s.solve(X)
    assert rc == 0
    for r in range(3):
        xo = o.solve(B[:, r])
        assert np.abs(X[:, r] - xo).max() <= FP64_X_TOL * np.abs(xo).max()


@pytest.mark.parametrize("nrhs", [8, 70])
def test_many_rhs_large_fronts(nrhs):
    """From 8 right-hand sides on, large fronts are solved with GEMM-shaped
    steps (RHS tiles of 64: 70 spans two tiles); every column matches the
    oracle's single-vector solve."""
    p = P.laplace3d(16)
    s = gpu_for(p, max_zero=1000)
    o = oracle_for(p, max_zero=1000)
    rng = np.random.default_rng(11)
    B = np.asfortranarray(rng.uniform(-1, 1, (p.n, nrhs)))
    X = B.copy(order="F")
    rep, rc = s.solve(X)
    assert rc == 0
    for r in (0, nrhs // 2, nrhs - 1):
        xo = o.solve(B[:, r])
        assert np.abs(X[:, r] - xo).max() <= FP64_X_TOL * np.abs(xo).max(), r
        assert P.backward_error(p.n, p.col, p.row, p.val, X[:, r], B[:, r]) <= FP64_BWD_TOL


@pytest.mark.parametrize("sfm", [32, 64, 96, 128])
@pytest.mark.parametrize("nrhs", [1, 3, 9])
def test_small_front_bins_against_oracle(sfm, nrhs):
    """small_front_max 32 .. 128 on a 3D Laplacian with relaxed supernodes
    routes fronts through every small-front kernel (warp factor, one-CTA
    factor with 8-column DMMA panels in both size variants, warp-per-front
    solves with 1..4 row slots, the one-pass backward for nf <= 32) next to
    the blocked large-front path; one, three (in-kernel RHS loop) and nine
    (one RHS per CTA row) right-hand sides against the oracle's FP64 solve."""
    p = P.laplace3d(14)
    s = gpu_for(p, max_zero=40, small_front_max=sfm)
    o = oracle_for(p, max_zero=40)
    rng = np.random.default_rng(sfm + nrhs)
    B = np.asfortranarray(rng.uniform(-1, 1, (p.n, nrhs)))
    X = B.copy(order="F")
    rep, rc = s.solve(X if nrhs > 1 else X[:, 0])
    assert rc == 0
    for r in range(nrhs):
        xo = o.solve(B[:, r])
        assert np.abs(X[:, r] - xo).max() <= FP64_X_TOL * np.abs(xo).max(), r
        assert P.backward_error(p.n, p.col, p.row, p.val, X[:, r], B[:, r]) <= FP64_BWD_TOL, r


def test_deterministic_replay():
    p = P.laplace3d(12)
    s = gpu_for(p, small_front_max=40)
    x1 = p.rhs.copy(); s.solve(x1)
    assert s.factorize(p.val) == 0
    x2 = p.rhs.copy(); s.solve(x2)
    assert np.array_equal(x1, x2)


def test_without_graphs_matches():
    p = P.laplace2d(30)
    s0 = gpu_for(p)
    s1 = gpu_for(p, use_graph=0)
    x0, x1 = p.rhs.copy(), p.rhs.copy()
    s0.solve(x0); s1.solve(x1)
    assert np.array_equal(x0, x1)


@pytest.mark.parametrize("nrhs", [1, 10])
def test_refinement_graph_matches_host_loop(nrhs):
    """FP32 + FP64 refinement as one graph with a device-side WHILE condition
    (the default) and as the host-driven loop (graphs off): the same sweeps
    in the same order stop at the same sweep with bit-identical solutions."""
    p = P.laplace3d(16)
    rng = np.random.default_rng(3)
    B = np.asfortranarray(rng.uniform(-1, 1, (p.n, nrhs)))
    out = []
    for ug in (1, 0):
        s = gpu_for(p, precision=H.MFD_PREC_FP32_IR, small_front_max=48, use_graph=ug)
        X = B.copy(order="F")
        rep, rc = s.solve(X if nrhs > 1 else X[:, 0])
        assert rc == 0 and rep.converged == 1 and rep.backward_error <= 1e-12
        out.append((X, rep.iterations, rep.backward_error))
        X2 = B.copy(order="F")                          # a second solve on the same handle
        s.solve(X2 if nrhs > 1 else X2[:, 0])
        assert np.array_equal(X, X2)
    assert np.array_equal(out[0][0], out[1][0])
    assert out[0][1] == out[1][1] and out[0][2] == out[1][2]


def test_not_positive_definite_reports_pivot():
    p = P.laplace2d(12)
    val = p.val.copy()
    diag_pos = p.col[:-1] - 1                  # diagonal entries come first in each column
    val[diag_pos[5]] = -4.0
    s = H.Solver.analyze(p.n, p.col, p.row, p.order)
    info = s.factorize(val)
    assert info > 0
    with pytest.raises(H.MfdError) as e:
        s.solve(p.rhs.copy())
    assert e.value.code == -6


# ---------------------------------------------------------------------------
# FP32 factor + FP64 iterative refinement
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("mk", [lambda: P.laplace3d(16), lambda: P.diffusion3d(12)], ids=["lap3d", "diff3d"])
def test_fp32_ir_reaches_1e12(mk):
    p = mk()
    s = gpu_for(p, precision=H.MFD_PREC_FP32_IR, small_front_max=64)
    x = p.rhs.copy()
    rep, rc = s.solve(x)
    assert rc == 0 and rep.converged == 1
    assert rep.iterations >= 1
    bwd = P.backward_error(p.n, p.col, p.row, p.val, x, p.rhs)
    assert bwd <= 1e-12, bwd
    xo = oracle_for(p).solve(p.rhs)
    assert np.abs(x - xo).max() <= 1e-8 * np.abs(xo).max()


@pytest.mark.parametrize("variant,tol", [(0, 3e-5), (2, 1e-2)], ids=["3xtf32", "1xtf32"])
def test_fp32_tensor_update_against_ffma(variant, tol):
    """The tcgen05 trailing update (0: 3xTF32, 2: 1xTF32) against the FFMA tiles
    (1) on the same FP32 factorization: largest fronts' panels agree to the
    TF32 rounding level, and refinement still reaches 1e-12."""
    p = P.laplace3d(14)
    ref = gpu_for(p, precision=H.MFD_PREC_FP32_IR, small_front_max=40, reserved=(1, 0, 0, 0, 0, 0, 0))
    tc = gpu_for(p, precision=H.MFD_PREC_FP32_IR, small_front_max=40, reserved=(variant, 0, 0, 0, 0, 0, 0))
    sym = oracle_for(p).symbolic()
    nc = np.diff(sym["node_ptr"]); nr = np.diff(sym["lptr"])
    for node in np.argsort(-(nc + nr))[:4] + 1:
        f = int(nc[node - 1] + nr[node - 1]), int(nc[node - 1])
        a, b = lower_panel(ref.front_panel(int(node)), *f), lower_panel(tc.front_panel(int(node)), *f)
        assert np.abs(a - b).max() <= tol * np.abs(a).max(), node
    x = p.rhs.copy()
    rep, rc = tc.solve(x)
    assert rc == 0 and rep.backward_error <= 1e-12


def _dense_lower_ccs(a):
    n = a.shape[0]
    ptr, rows, vals = [1], [], []
    for j in range(n):
        rows.extend(range(j + 1, n + 1))
        vals.extend(a[j:, j])
        ptr.append(len(rows) + 1)
    return np.array(ptr, np.int32), np.array(rows, np.int32), np.array(vals, np.float64)


@pytest.mark.parametrize("small", [1e-4, None], ids=["small_pivot", "no_small_pivot"])
def test_fp32_potrf_small_pivot_falls_back_to_fp64(small):
    """The FP32 factorization's diagonal blocks run their pivot chain in FP32
    and redo a 32-column sub-block in FP64 when a pivot falls below 2^-12 of
    the diagonal entry it started from.  A dense SPD front A = L diag(d) L^T
    (n = 300: one front, three 128-column panel steps on the blocked path)
    whose pivot 41 is d_41 = 1e-4 x its column's scale triggers the fallback;
    refinement reaches 1e-12, and x matches the FP64 solution within
    10 cond(A) times the refinement tolerance (the forward error a solution
    with backward error 1e-12 can have).  Without the small pivot no
    sub-block falls back."""
    n = 300
    rng = np.random.default_rng(8)
    L = np.tril(rng.uniform(-0.3, 0.3, (n, n)), -1) + np.eye(n)
    d = rng.uniform(1.0, 2.0, n)
    if small is not None:
        d[40] = small
    A = (L * d) @ L.T
    col, row, val = _dense_lower_ccs(A)
    s = H.Solver.analyze(n, col, row, None, max_zero=0, precision=H.MFD_PREC_FP32_IR)
    assert s.stats().num_front == 1 and s.stats().max_front == n
    assert s.factorize(val) == 0
    fb = s.stats().pivot_fallbacks
    assert (fb >= 1) if small is not None else (fb == 0), fb
    xt = rng.uniform(-1, 1, n)
    b = A @ xt
    x = b.copy()
    rep, rc = s.solve(x)
    assert rc == 0 and rep.converged == 1 and rep.backward_error <= 1e-12
    xr = np.linalg.solve(A, b)
    assert np.abs(x - xr).max() <= 10 * np.linalg.cond(A) * 1e-12 * np.abs(xr).max()
    s64 = H.Solver.analyze(n, col, row, None, max_zero=0)
    assert s64.factorize(val) == 0 and s64.stats().pivot_fallbacks == 0


@pytest.mark.parametrize("k", [10, 37])
def test_fp32_ir_many_rhs(k):
    """Block refinement: all right-hand sides refined together (residuals of
    all columns in one multi-column SpMV: 37 columns take two 32-lane passes
    and a partial transpose tile), each column to backward error <= 1e-12."""
    p = P.laplace3d(16)
    s = gpu_for(p, max_zero=1000, precision=H.MFD_PREC_FP32_IR)
    rng = np.random.default_rng(5)
    B = np.asfortranarray(rng.uniform(-1, 1, (p.n, k)))
    X = B.copy(order="F")
    rep, rc = s.solve(X)
    assert rc == 0 and rep.converged == 1
    for r in range(k):
        assert P.backward_error(p.n, p.col, p.row, p.val, X[:, r], B[:, r]) <= 1e-12, r


# ---------------------------------------------------------------------------
# batch of independent systems (uneven sizes)
# ---------------------------------------------------------------------------
def test_batch_uneven():
    probs = P.laplace2d_batch(count=12, seed=3, lo=8, hi=40)
    s = H.Solver.analyze_batch([(q.n, q.col, q.row, q.order) for q in probs])
    a = np.concatenate([q.val for q in probs])
    assert s.factorize(a) == 0
    b = np.concatenate([q.rhs for q in probs])
    x = b.copy()
    rep, rc = s.solve(x)
    assert rc == 0
    off = 0
    for i, q in enumerate(probs):
        o = O.Oracle.analyze(q.n, q.col, q.row, nb=10, max_zero=10, order_perm=q.order)
        assert o.factorize(q.val) == 0
        xo = o.solve(q.rhs)
        xi = x[off:off + q.n]
        assert np.abs(xi - xo).max() <= FP64_X_TOL * np.abs(xo).max(), i
        # per-system device index data equals the oracle's
        assert np.array_equal(s.index(H.LOCAL_INDEX, i), o.get(O.LOCAL))
        off += q.n


# ---------------------------------------------------------------------------
# the reference-named API on the reference's own end-to-end fixtures
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("name", ["bcsstk01.mtx", "poisson_9_9.mtx"])
def test_hppllt_api_fixture(name):
    from test_oracle_e2e import coo_to_ccs, sym_matvec
    m = json.load(open(os.path.join(HERE, "golden", "mtx_fixtures.json")))[name]
    n = m["n"]
    ptr, row, val = coo_to_ccs(n, m["row"], m["col"], m["val"])
    H.hppllt_init(R.HPPLLT_TEST_OPTIONS)
    H.hppllt_analyze(ptr, row, n)
    assert H.hppllt_factorize(val) == 0
    b = np.full(n, 10.0)
    H.hppllt_solve(b)
    r = 10.0 - sym_matvec(n, ptr, row, val, b)
    assert np.linalg.norm(r) / np.linalg.norm(b) <= R.HPPLLT_TEST_TOL
    assert H.hppllt_get_cost() > 0 and H.hppllt_get_nonzero() > 0
    o = O.Oracle.analyze(n, ptr, row, nb=10, max_zero=10)
    assert H.hppllt_get_cost() == o.cost()
    assert H.hppllt_get_nonzero() == o.nonzero()           # count_nonzero (cost_calculator_m.f90:22-33)
    for k in (1, 2, 3):
        assert H.hppllt_get_array_size(k) == o.array_size(k)
    H.hppllt_finalize()
