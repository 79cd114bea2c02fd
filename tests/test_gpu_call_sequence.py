"""A handle's first factorization and its first solve of a kind are launched directly, the second ones captured as
graphs, the later ones replayed: whichever a call is, it gives the same bits for the same values, also when the
values, the right-hand sides or their number change from one to the next."""
import numpy as np
import pytest

from mfdag import hppllt as H
from mfdag import problems as P

pytestmark = pytest.mark.gpu


def _handle(kind, **opts):
    if kind == "batch":
        ps = list(P.laplace2d_batch(12, lo=16, hi=40))
        s = H.Solver.analyze_batch([(p.n, p.col, p.row, p.order) for p in ps], max_zero=100, **opts)
        val = np.concatenate([p.val for p in ps])
    else:
        p = P.laplace3d(14)
        s = H.Solver.analyze(p.n, p.col, p.row, p.order, max_zero=1000, small_front_max=48, **opts)
        val = np.array(p.val)
    return s, val


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["laplace", "batch"])
def test_first_captured_and_replayed_calls_agree(kind, precision):
    s, val = _handle(kind, precision=precision)
    rng = np.random.default_rng(5)
    vals = [val, 1.5 * val, 0.75 * val]                  # other values, still positive definite
    B = np.asfortranarray(rng.uniform(-1, 1, (s.n, 9)))
    want = {}
    for v, a in enumerate(vals):                         # a handle without graphs for each
        r, _ = _handle(kind, precision=precision, use_graph=0)
        assert r.factorize(a) == 0
        for k in (1, 3, 9):
            X = B[:, :k].copy(order="F")
            rep, rc = r.solve(X)
            assert rc == 0
            want[v, k] = (X, rep.iterations, rep.backward_error)
        r.close()
    for v in (0, 1, 2, 0, 1):                            # factorizations 1 .. 5
        assert s.factorize(vals[v]) == 0
        for k in (1, 3, 9, 3, 1, 1):                     # storage grows twice in the first round
            for report in (True, False):
                X = B[:, :k].copy(order="F")
                rep, rc = s.solve(X, report=report)
                assert rc == 0
                assert np.array_equal(X, want[v, k][0]), (v, k, report)
                if report:
                    assert rep.iterations == want[v, k][1]
                    assert rep.backward_error <= 1.01 * want[v, k][2] + 1e-18
                    assert 0 < rep.time_ms < 1000
    s.close()


def test_device_times_leave_the_capture_out():
    """factor_ms and time_ms are the device's: those of the captured call lie with those of the replays."""
    s, val = _handle("laplace")
    b = np.random.default_rng(1).uniform(-1, 1, s.n)
    f, t = [], []
    for _ in range(6):
        assert s.factorize(val) == 0
        f.append(s.stats().factor_ms)
        rep, rc = s.solve(b.copy())
        t.append(rep.time_ms)
    assert f[1] <= 3 * np.median(f[2:]) + 0.2 and t[1] <= 3 * np.median(t[2:]) + 0.2
    s.close()


def test_handles_on_several_threads():
    """Four threads, each with handles of its own coming and going: direct first calls, captures, replays, set-ups and
    frees of one thread run while the others capture.  Every solution has the bits of a handle used alone."""
    import threading
    kinds = [("laplace", 0), ("batch", 0), ("laplace", 1), ("batch", 1)]
    alone = {}
    for kind, precision in kinds:
        s, val = _handle(kind, precision=precision)
        b = np.random.default_rng(9).uniform(-1, 1, s.n)
        assert s.factorize(val) == 0
        x = b.copy()
        s.solve(x)
        alone[kind, precision] = x
        s.close()
    errors = []

    def work(first):
        try:
            for turn in range(6):
                kind, precision = kinds[(first + turn) % 4]
                s, val = _handle(kind, precision=precision)
                b = np.random.default_rng(9).uniform(-1, 1, s.n)
                for _ in range(4):
                    assert s.factorize(val) == 0
                    x = b.copy()
                    rep, rc = s.solve(x)
                    assert rc == 0 and np.array_equal(x, alone[kind, precision])
                s.close()
        except BaseException as e:                       # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not errors and not any(t.is_alive() for t in threads), errors
