"""The work that programs have this solver do, as sized cases with their inputs.

A program analyses a sparsity pattern once, keeps the handle, and then
factorizes new values on it and solves (a Newton or time step, a parameter
sweep), or factorizes once and solves many right-hand sides (implicit time
stepping with a constant matrix).  Both are here, through the handle API of
mfdag.hppllt, with values and right-hand sides in device memory.  Kinds:

  lap2d    5-point Laplacian plus a small random diagonal shift, 2D grid
  lap3d    7-point Laplacian plus a small random diagonal shift, 3D grid
  diff3d   7-point diffusion, per-cell conductivities 10^U[-2, 2]
  elast    Q1 hexahedral elasticity, 3 dofs per node, one face clamped
  batch    count square lap2d systems, sides uniform in [nx, ny], held by one handle

``mixed`` selects the FP32 factor with FP64 refinement (to a backward error of
1e-12).  ``what`` is "step" (factorize, then solve) or "solve" (the factor is
at hand).  Every right-hand side is b = A x* for an x* drawn from U[-1, 1],
so x* is the value that a pass returns.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multifrontal-dag_b200"))

from mfdag import hppllt as H  # noqa: E402
from mfdag import problems as P  # noqa: E402

# relaxed-supernode threshold that the benchmark uses for each kind
MAX_ZERO = {"lap2d": 10, "lap3d": 1000, "diff3d": 1000, "elast": 1000, "batch": 100}


def _case(name, kind, nx, ny=0, nz=0, what="step", mixed=False, nrhs=1, count=1):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "what": what, "mixed": mixed, "nrhs": nrhs, "count": count}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a coarse 2D model refactorized and solved inside another loop; all latency
        _case("lap2d_17x19_step", "lap2d", 17, 19),
        # a plain 2D solver run, 100 x 100
        _case("lap2d_100x100_step", "lap2d", 100, 100),
        # implicit time stepping on a kept factor, one right-hand side a step, odd sizes
        _case("lap3d_37x41x43_solve", "lap3d", 37, 41, 43, what="solve"),
        # a 3D run at scale in FP64: top fronts of about 4,000 columns
        _case("lap3d_64_step", "lap3d", 64, 64, 64),
        # the same run with the FP32 factor and FP64 refinement
        _case("lap3d_64_mixed_step", "lap3d", 64, 64, 64, mixed=True),
        # an ordinary FP64 3D model with a strongly varying coefficient, a handful of load cases
        _case("diff3d_30x33x35_5rhs_step", "diff3d", 30, 33, 35, nrhs=5),
        # the largest single system: variable-coefficient diffusion, mixed precision
        _case("diff3d_80_mixed_step", "diff3d", 80, 80, 80, mixed=True),
        # structural model with 64 load cases, FP64
        _case("elast_30_64rhs_step", "elast", 30, 30, 30, nrhs=64),
        # a smaller structural model, mixed precision, 16 load cases
        _case("elast_21_mixed_16rhs_step", "elast", 21, 21, 21, mixed=True, nrhs=16),
        # many uneven independent systems in one handle, FP64
        _case("batch_1000_step", "batch", 16, 128, count=1000),
        # a smaller batch, mixed precision
        _case("batch_300_mixed_step", "batch", 16, 128, mixed=True, count=300),
        # the kept factors of a batch, one right-hand side each
        _case("batch_200_solve", "batch", 16, 128, what="solve", count=200),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lap2d", "lap3d", "diff3d", "elast", "batch"])
    mixed = rng.random() < 0.4
    what = "solve" if rng.random() < 0.35 else "step"
    nrhs = rng.choice([1, 1, 1, rng.randint(2, 7), rng.randint(8, 64)])
    if kind == "lap2d":
        s = _log(rng, 16, 200)
        return _case("", kind, s, max(16, s + rng.randint(-5, 5)), 0, what, mixed, nrhs)
    if kind == "batch":
        lo = rng.randint(16, 40)
        return _case("", kind, lo, rng.randint(lo + 20, 128), 0, what, mixed, 1, _log(rng, 30, 500))
    if kind == "elast":
        return _case("", kind, _log(rng, 6, 24), _log(rng, 6, 24), _log(rng, 6, 24), what, mixed, nrhs)
    s = _log(rng, 12, 52)
    return _case("", kind, s, max(10, s + rng.randint(-4, 4)), max(10, s + rng.randint(-4, 4)), what, mixed, nrhs)


# ---- patterns (host, the same for every seed) -------------------------------------
@functools.lru_cache(maxsize=None)
def _grid(dims, dof=1):
    """Lower CCS of the 5- or 7-point pattern (x fastest; a column's rows ascending, the
    diagonal first), which of a cell's candidate entries exist, and the ordering."""
    n = int(np.prod(dims))
    coords = np.unravel_index(np.arange(n), dims[::-1])[::-1]
    strides = np.cumprod((1,) + dims[:-1])
    mask = np.stack([np.ones(n, bool)] + [coords[a] < d - 1 for a, d in enumerate(dims)], axis=1)
    row = np.stack([np.arange(n)] + [np.arange(n) + s for s in strides], axis=1)[mask] + 1
    ptr = np.concatenate([[1], 1 + np.cumsum(mask.sum(axis=1))])
    return n, ptr.astype(np.int32), row.astype(np.int32), mask, P.nested_dissection(dims)


@functools.lru_cache(maxsize=None)
def _elast(ne):
    """Pattern of the clamped Q1 elasticity matrix on an ne[0] x ne[1] x ne[2] element mesh:
    lower CCS, ordering, and each element entry's place among the matrix's entries."""
    ex, ey, ez = (v.ravel() for v in np.meshgrid(*(np.arange(k) for k in ne), indexing="ij"))
    nx, ny, nz = ne[0], ne[1] + 1, ne[2] + 1                      # free nodes: x = 1 .. ne[0]
    n = 3 * nx * ny * nz
    gd = np.empty((ex.size, 24), np.int64)
    for k in range(8):
        a, b, c = k & 1, k >> 1 & 1, k >> 2
        node = (ex + a - 1) + nx * ((ey + b) + ny * (ez + c))
        for d in range(3):
            gd[:, 3 * k + d] = np.where(ex + a >= 1, 3 * node + d, -1)
    r, c = np.repeat(gd, 24, axis=1), np.tile(gd, (1, 24))        # element entry 24 i + j: row i, column j
    keep = (r >= c) & (c >= 0)
    key, place = np.unique(c[keep] * n + r[keep], return_inverse=True)
    col, row = key // n, key % n
    ptr = np.concatenate([[1], 1 + np.cumsum(np.bincount(col, minlength=n))])
    order = P.nested_dissection((nx, ny, nz), dof=3)
    # the whole symmetric matrix, rows padded to the longest, for b = A x*
    off = row != col
    fr = np.concatenate([row, col[off]])
    fc = np.concatenate([col, row[off]])
    src = np.concatenate([np.arange(key.size), np.nonzero(off)[0]])
    o = np.lexsort((fc, fr))
    fr, fc, src = fr[o], fc[o], src[o]
    cnt = np.bincount(fr, minlength=n)
    slot = np.arange(fr.size) - np.repeat(np.cumsum(cnt) - cnt, cnt)
    ell_c = np.zeros((n, cnt.max()), np.int64)
    ell_s = np.full((n, cnt.max()), key.size, np.int64)           # one past the end: a zero value
    ell_c[fr, slot], ell_s[fr, slot] = fc, src
    e, i = np.nonzero(keep)
    return n, ptr.astype(np.int32), (row + 1).astype(np.int32), order, (e, i, place.ravel()), (ell_c, ell_s)


@functools.lru_cache(maxsize=None)
def _sides(lo, hi, count):
    return tuple(int(s) for s in np.random.default_rng(3).integers(lo, hi + 1, size=count))


@functools.lru_cache(maxsize=None)
def _elast_parts():
    return tuple(k.ravel() for k in P._hex_stiffness_parts())


def _systems(case):
    """(n, ccs_col, ccs_row, order) of every system of the case."""
    if case["kind"] == "batch":
        return [(g[0], g[1], g[2], g[4]) for g in (_grid((s, s)) for s in _sides(case["nx"], case["ny"], case["count"]))]
    if case["kind"] == "elast":
        g = _elast((case["nx"], case["ny"], case["nz"]))
        return [g[:4]]
    g = _grid(_dims(case))
    return [(g[0], g[1], g[2], g[4])]


def _dims(case):
    return (case["nx"], case["ny"]) if case["kind"] == "lap2d" else (case["nx"], case["ny"], case["nz"])


# ---- values ---------------------------------------------------------------------------
def _grid_values(entries, mask):
    """The columns' candidate entries (diagonal, then one per axis) that exist, in CCS order."""
    return torch.stack(entries, dim=1)[torch.from_numpy(mask).cuda()]


def _stencil(diag, faces, x, dims):
    """A x for A = diag(diag) plus, per axis, the couplings faces[a] to the next cell."""
    shape = dims[::-1]
    y = (diag * x).view(shape)
    xv = x.view(shape)
    for a in range(len(dims)):
        ax, m = len(dims) - 1 - a, dims[a] - 1
        f = faces[a].view(shape).narrow(ax, 0, m)
        y.narrow(ax, 0, m).add_(f * xv.narrow(ax, 1, m))
        y.narrow(ax, 1, m).add_(f * xv.narrow(ax, 0, m))
    return y.reshape(-1)


def _x_true(case, seed):
    n = sum(s[0] for s in _systems(case))
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 2 + 1)
    return torch.rand((case["nrhs"], n), generator=g, dtype=torch.float64, device="cuda") * 2 - 1


def _laplace(dims, shift):
    """Diagonal and couplings of the Laplacian with shift[i] added to the diagonal."""
    return 2.0 * len(dims) + shift, [torch.full_like(shift, -1.0) for _ in dims]


def _diffusion(dims, k):
    """Diagonal and couplings of the diffusion matrix with cell conductivities k: a face carries the
    harmonic mean, a boundary face adds twice its cell's to the diagonal."""
    shape = dims[::-1]
    kv, diag, faces = k.view(shape), torch.zeros(shape, dtype=k.dtype, device=k.device), []
    for a in range(len(dims)):
        ax, m = len(dims) - 1 - a, dims[a] - 1
        lo, hi = kv.narrow(ax, 0, m), kv.narrow(ax, 1, m)
        f = 2.0 * lo * hi / (lo + hi)
        diag.narrow(ax, 0, 1).add_(2.0 * kv.narrow(ax, 0, 1))
        diag.narrow(ax, m, 1).add_(2.0 * kv.narrow(ax, m, 1))
        diag.narrow(ax, 0, m).add_(f)
        diag.narrow(ax, 1, m).add_(f)
        full = torch.zeros_like(diag)
        full.narrow(ax, 0, m).copy_(-f)
        faces.append(full.reshape(-1))
    return diag.reshape(-1), faces


def _values(case, seed, x):
    """The matrix's values in CCS order and b = A x, in device memory."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 2)

    def rand(n):
        return torch.rand(n, generator=g, dtype=torch.float64, device="cuda")

    if case["kind"] == "batch":
        sides = _sides(case["nx"], case["ny"], case["count"])
        shift = (0.1 * rand(len(sides))).tolist()
        vals, rhs, at = [], [], 0
        for s, sh in zip(sides, shift):
            diag, faces = _laplace((s, s), torch.full((s * s,), sh, dtype=torch.float64, device="cuda"))
            vals.append(_grid_values([diag] + faces, _grid((s, s))[3]))
            rhs.append(_stencil(diag, faces, x[0, at:at + s * s], (s, s)))
            at += s * s
        return torch.cat(vals), torch.cat(rhs)[None]
    if case["kind"] == "elast":
        n, _, row, _, (e, i, place), (ell_c, ell_s) = _elast((case["nx"], case["ny"], case["nz"]))
        nel = case["nx"] * case["ny"] * case["nz"]
        young, nu = (10.0 ** (2.0 * rand(nel) - 1.0)).cpu().numpy(), (0.25 + 0.1 * rand(nel)).cpu().numpy()
        lam, mu = young * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), young / (2.0 * (1.0 + nu))
        kl, km = _elast_parts()
        val = torch.from_numpy(np.bincount(place, weights=lam[e] * kl[i] + mu[e] * km[i], minlength=row.size)).cuda()
        full = torch.cat([val, val.new_zeros(1)])[torch.from_numpy(ell_s).cuda()]
        cols = torch.from_numpy(ell_c).cuda()
        return val, torch.stack([(full * v[cols]).sum(dim=1) for v in x])
    dims = _dims(case)
    n, _, _, mask, _ = _grid(dims)
    diag, faces = _diffusion(dims, 10.0 ** (4.0 * rand(n) - 2.0)) if case["kind"] == "diff3d" else _laplace(dims, 0.1 * rand(n))
    return _grid_values([diag] + faces, mask), torch.stack([_stencil(diag, faces, v, dims) for v in x])


# ---- a pass ---------------------------------------------------------------------------
def prepare(case, seed):
    x = _x_true(case, seed)
    a, b = _values(case, seed, x)
    a, b = a.contiguous(), b.contiguous()
    opts = {"max_zero": MAX_ZERO[case["kind"]], "precision": H.MFD_PREC_FP32_IR if case["mixed"] else H.MFD_PREC_FP64}
    systems = _systems(case)
    solver = H.Solver.analyze_batch(systems, **opts) if case["kind"] == "batch" else H.Solver.analyze(*systems[0], **opts)
    torch.cuda.synchronize()
    if case["what"] == "solve" and solver.factorize(a) != 0:
        raise RuntimeError("the matrix is not positive definite")
    return {"solver": solver, "a": a, "b": b, "nrhs": case["nrhs"], "step": case["what"] == "step"}


def run(state):
    solver = state["solver"]
    x = state["b"].clone()
    if state["step"] and solver.factorize(state["a"]) != 0:
        raise RuntimeError("the matrix is not positive definite")
    # solve() works on the handle's own stream: what wrote x on this one has to be done first
    torch.cuda.current_stream().synchronize()
    _, rc = solver.solve(x, nrhs=state["nrhs"])
    if rc != 0:
        raise RuntimeError(f"solve returned {rc}")
    return x


@functools.lru_cache(maxsize=None)
def _counts(n, col, row, order, max_zero):
    s = H.symbolic_analyze(n, np.frombuffer(col, np.int32), np.frombuffer(row, np.int32), np.frombuffer(order, np.int32),
                           max_zero)
    nc = np.diff(s["node_ptr"]).astype(np.float64)
    nr = np.diff(s["lptr"]).astype(np.float64)

    def sq(k):
        return k * (k + 1) * (2 * k + 1) / 6

    return float((sq(nr + nc) - sq(nr)).sum()), float((nc * nr + nc * (nc + 1) / 2).sum())


def work(case):
    """Factorization: each value of A read and each entry of the factor written once, sum k^2
    operations over its columns; solve: each entry of the factor read once, four operations per
    entry and right-hand side; each right-hand side read and each solution written once."""
    flops = size = values = n = 0.0
    for s in _systems(case):
        f, z = _counts(s[0], s[1].tobytes(), s[2].tobytes(), s[3].tobytes(), MAX_ZERO[case["kind"]])
        flops, size, values, n = flops + f, size + z, values + s[2].size, n + s[0]
    w = 4.0 if case["mixed"] else 8.0
    vectors, solve = 16.0 * n * case["nrhs"], 4.0 * size * case["nrhs"]
    if case["what"] == "solve":
        return {"bytes": w * size + vectors, "flops": solve}
    return {"bytes": 8.0 * values + w * size + vectors, "flops": flops + solve}


def exact(case, seed):
    return _x_true(case, seed)
