"""Which launch of its level a small front goes to (csrc/small_bins.hpp), compiled on its own with checked
vector indexing: every front up to the handle's line gets a bin that exists and is large enough for it, the
others none, whatever the line (small_front_max takes any positive value) and whatever else is on the level."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multifrontal-dag_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "small_bins.hpp"
int main(int argc, char** argv) {              // line, then the level's front orders
  const int sfm = std::atoi(argv[1]);
  std::vector<int> orders;
  for (int i = 2; i < argc; ++i) orders.push_back(std::atoi(argv[i]));
  const std::vector<int> bins = mfd::small_bin_sizes(sfm), of = mfd::small_bins_of_level(bins, sfm, orders);
  for (int b : bins) std::printf("%d ", b);
  std::printf("\n");
  for (int b : of) std::printf("%d ", b);
  std::printf("\n");
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("small_bins")
    (d / "main.cpp").write_text(PROGRAM)
    exe = str(d / "main")
    subprocess.run(["g++", "-std=c++17", "-O1", "-D_GLIBCXX_ASSERTIONS", "-I", CSRC, str(d / "main.cpp"), "-o", exe], check=True)
    return exe


LEVELS = [[10, 30], [1, 2, 8, 9, 16, 17, 24, 25, 31, 32, 33, 64, 65, 128, 160, 161, 400], [30] * 3553, [12] * 3553 + [30]]


@pytest.mark.parametrize("line", [1, 8, 15, 16, 17, 23, 24, 31, 32, 33, 40, 96, 100, 160])
@pytest.mark.parametrize("level", range(len(LEVELS)))
def test_every_small_front_has_a_bin(program, line, level):
    orders = LEVELS[level]
    r = subprocess.run([program, str(line)] + [str(n) for n in orders], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    bins, of = ([int(v) for v in row.split()] for row in r.stdout.splitlines()[:2])
    assert bins == sorted(set(bins)) and bins[-1] == line
    for n, b in zip(orders, of):
        if n > line:
            assert b == -1
        else:
            assert 0 <= b < len(bins) and n <= bins[b]
            assert n <= 32 or b == 0 or bins[b - 1] < n          # above one warp: the narrowest that holds it


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("line", [1, 8, 16, 24, 31])
def test_lines_below_one_warp_against_oracle(line, precision):
    """A 2D Laplacian with relaxed supernodes, whose levels mix fronts on both sides of the line, one and three
    right-hand sides, against the oracle's FP64 solve.  The condition number is below 300: both solves in FP64,
    1e-10; FP32 + refinement to a backward error of 1e-12, 1e-9."""
    import numpy as np
    from mfdag import hppllt as H
    from mfdag import problems as P
    from oracle import oracle as O
    p = P.laplace2d(23)
    o = O.Oracle.analyze(p.n, p.col, p.row, nb=10, max_zero=10, order_perm=p.order)
    assert o.factorize(p.val) == 0
    s = H.Solver.analyze(p.n, p.col, p.row, p.order, max_zero=10, small_front_max=line, precision=precision)
    assert s.factorize(p.val) == 0
    B = np.asfortranarray(np.random.default_rng(line).uniform(-1, 1, (p.n, 3)))
    for X in (B[:, 0].copy(), B.copy(order="F")):
        rep, rc = s.solve(X)
        assert rc == 0
        for r, x in enumerate(X.reshape(p.n, -1).T):
            xo = o.solve(B[:, r])
            assert np.abs(x - xo).max() <= (1e-10 if precision == 0 else 1e-9) * np.abs(xo).max()
            assert P.backward_error(p.n, p.col, p.row, p.val, x, B[:, r]) <= 1e-12
