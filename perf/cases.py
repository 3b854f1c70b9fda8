"""Performance cases: the calls a user of the multifrontal library makes, over
the sizes, precisions and options they are made with.

A case is one pass through the public entry points of `mfgpu` on a handle that
is kept between passes, as a time-stepping, Newton or design loop keeps it:

  op = "solve"    right-hand sides against a kept factorization
       "apply"    the factored operator applied to vectors (the check of a
                  factorization, or a matrix-free product)
       "factor"   new matrix values, full factorization, solve
       "update"   coefficients of a small box changed: localized update, solve
       "step"     full factorization, localized update, solve
       "batch"    independent 2D problems in one handle: full factorization
                  and solve of all of them

`host` cases pass numpy vectors through Solve(), the others device buffers.
Grids, coefficient ranges, leaf parameters and right-hand-side counts are those
of the benchmark and the tests, or of the same kind.  Mixed precision refines to
a relative residual of 1e-12, about what the FP64 path reaches.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "updating-multifrontal_b200"))

import mfgpu  # noqa: E402
from mfgpu import stencil  # noqa: E402

REFINE_TOL = 1e-12
PATCH = {2: 9, 3: 5}          # cells a side of the box whose coefficients an update changes
PATCH_FACTOR = 10.0


def _case(op, N, name=None, precision="fp64", nrhs=1, width=1, leaf=4, lo=0.1, hi=10.0, at=0.37,
          host=False):
    """A single-problem case; N has two or three grid sizes, `at` places the
    changed box of an update along every axis (0 .. 1)."""
    c = {"op": op, "nx": int(N[0]), "ny": int(N[1]), "nz": int(N[2]) if len(N) == 3 else 0,
         "precision": precision, "nrhs": int(nrhs), "width": int(width), "leaf": int(leaf),
         "lo": float(lo), "hi": float(hi), "at": float(at), "host": bool(host)}
    return dict(c, name=name) if name else c


def _batch(sides, name=None, nrhs=4, precision="fp64", leaf=4):
    c = {"op": "batch", "sides": " ".join(str(s) for s in sides), "precision": precision,
         "nrhs": int(nrhs), "leaf": int(leaf), "lo": 0.1, "hi": 10.0}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one right-hand side from a host program against a small kept factorization: the call
        # of an interactive or embedded user, latency only
        _case("solve", (63, 63), "solve-2d-63-host", host=True),
        # the CPU-sized 2D problem of the benchmark: a whole step is a few hundred small fronts
        _case("step", (127, 127), "step-2d-127"),
        # the benchmark's large 2D problem: new coefficients, factorization, 4 right-hand sides
        _case("factor", (1023, 1023), "factor-2d-1023", nrhs=4, leaf=8),
        # the same grid in a design loop: a 9 x 9 patch changes, everything else is kept
        _case("update", (1023, 1023), "update-2d-1023", nrhs=4, leaf=8),
        # the factored operator applied to a few vectors
        _case("apply", (511, 511), "apply-2d-511", nrhs=4, leaf=8),
        # a fourth-order (wider, nonsymmetric) stencil, factored by pivoted LU
        _case("factor", (127, 127), "wide-2d-127", width=2, lo=0.5, hi=2.0),
        # a ragged 2D grid in mixed precision: the tree's last leaf boxes take what the others leave
        _case("factor", (700, 333), "factor-2d-700x333-mixed", precision="mixed", nrhs=2, leaf=8),
        # many right-hand sides (sources, columns of an inverse) on a kept 3D factorization
        _case("solve", (63, 63, 63), "solve-3d-63-rhs16", nrhs=16, hi=100.0),
        # a mid-sized 3D problem in mixed precision
        _case("factor", (63, 63, 63), "factor-3d-63-mixed", precision="mixed", hi=100.0),
        # a ragged 3D grid, plain FP64
        _case("factor", (79, 63, 50), "factor-3d-79x63x50", hi=100.0),
        # the serving-sized 3D problem, mixed precision: factorization, localized update, solve
        _case("step", (95, 95, 95), "step-3d-95-mixed", precision="mixed"),
        # independent 2D problems of uneven sizes in one handle
        _batch([63] * 10 + [127] * 8 + [255] * 4 + [191, 100], "batch-2d-24"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _divides(case):
    """Whether the tree's leaf boxes come out non-empty on this grid (long, thin ones may not)."""
    probs = [(2, (m, m), 1) for m in _sides(case)] if case["op"] == "batch" else \
        [(len(_grid(case)), _grid(case), case["width"])]
    try:
        for dim, N, width in probs:
            mfgpu.Symbolic(dim, N, width, case["leaf"])
    except RuntimeError:
        return False
    return True


def draw(rng):
    """One more case of the listed ones' ranges."""
    while True:
        case = _draw(rng)
        if _divides(case):
            return case


def _draw(rng):
    kind = rng.choice(["2d-small", "2d-large", "3d", "3d", "wide", "batch"])
    if kind == "batch":
        return _batch([_log_int(rng, 40, 255) for _ in range(rng.randint(6, 24))],
                      nrhs=rng.randint(1, 8), precision=rng.choice(["fp64", "mixed"]))
    if kind == "wide":
        return _case(rng.choice(["factor", "step", "solve"]),
                     (_log_int(rng, 31, 127), _log_int(rng, 31, 127)), width=rng.choice([2, 3]),
                     nrhs=rng.randint(1, 4), lo=0.5, hi=2.0, at=rng.random())
    op = rng.choice(["solve", "apply", "factor", "update", "step"])
    nrhs = _log_int(rng, 1, 16) if op in ("solve", "apply") else rng.randint(1, 4)
    host = op == "solve" and rng.random() < 0.3
    # (the mixed path's factored operator is an FP32 one: applying it is a diagnostic)
    precision = "fp64" if op == "apply" else rng.choice(["fp64", "mixed"])
    if kind == "3d":
        while True:
            N = [_log_int(rng, 20, 95) for _ in range(3)]
            # the cost goes with the sixth power of the side: FP64 stays below the listed ragged
            # grid's, mixed below the 95^3 step's
            if math.prod(N) ** (1 / 3) <= (62 if precision == "fp64" else 90) and \
                    max(N) <= 3 * min(N):
                break
        return _case(op, N, precision=precision, nrhs=nrhs, hi=rng.choice([10.0, 100.0]),
                     at=rng.random(), host=host)
    r, leaf = ((31, 255), rng.choice([4, 8])) if kind == "2d-small" else ((256, 1023), 8)
    N = [_log_int(rng, *r) for _ in range(2)]
    return _case(op, N, precision=precision, nrhs=nrhs, leaf=leaf, at=rng.random(), host=host)


def _grid(case):
    return (case["nx"], case["ny"]) + ((case["nz"],) if case["nz"] else ())


def _sides(case):
    return [int(s) for s in case["sides"].split()]


def _patch(case):
    """Lower corner and side of the box of cells that an update changes."""
    N = _grid(case)
    side = min(PATCH[len(N)], min(N))
    return [int(case["at"] * (n - side)) for n in N], side


def _coefficients(case, N, seed):
    w = case.get("width", 1)
    rng = np.random.Generator(np.random.PCG64(seed))
    u = rng.random(tuple(n + 2 * w for n in N))
    return case["lo"] * np.power(case["hi"] / case["lo"], u)


def _changed(case, a):
    lo, side = _patch(case)
    w = case["width"]
    a2 = a.copy()
    a2[tuple(slice(l + w, l + w + side) for l in lo)] *= PATCH_FACTOR
    return a2


def _rhs(case, n, seed):
    rng = np.random.Generator(np.random.PCG64(seed + 7919))
    return rng.uniform(-1.0, 1.0, (case["nrhs"], n))


def prepare(case, seed):
    kw = dict(precision=mfgpu.MFGPU_MIXED if case["precision"] == "mixed" else mfgpu.MFGPU_FP64,
              refine_tol=REFINE_TOL)
    op = case["op"]
    if op == "batch":
        mats = [(stencil.build_laplacian(_coefficients(case, (m, m), seed * 1000 + i)), (m, m), 1,
                 case["leaf"]) for i, m in enumerate(_sides(case))]
        F = mfgpu.MFBatch(mats, **kw)
        A, A2, mod = F.A, None, None
    else:
        N, w = _grid(case), case["width"]
        a = _coefficients(case, N, seed)
        A, A2, mod = stencil.build_laplacian(a, width=w), None, None
        F = (mfgpu.MF2D if len(N) == 2 else mfgpu.MF3D)(A, *N, w, case["leaf"], **kw)
        if op in ("update", "step"):
            A2 = stencil.build_laplacian(_changed(case, a), width=w)
            mod = stencil.modified_dofs(A, A2)
    b = _rhs(case, A.n, seed)
    s = {"op": op, "host": case.get("host", False), "F": F, "n": A.n, "nnz": A.nnz,
         "nrhs": case["nrhs"], "mod": mod, "val": torch.from_numpy(A.val).cuda(),
         "val2": torch.from_numpy(A2.val).cuda() if A2 is not None else None}
    if s["host"]:
        s["b"] = np.asfortranarray(b.T)
    else:
        s["b"] = torch.from_numpy(b).cuda()
        s["x"] = torch.empty_like(s["b"])
    torch.cuda.synchronize()       # the handle works on a stream of its own
    if op in ("solve", "apply", "update"):
        F.Factor()
    return s


def run(s):
    F, op, n, nrhs = s["F"], s["op"], s["n"], s["nrhs"]
    if op in ("factor", "step", "batch"):
        F.refactor_device(s["val"].data_ptr(), s["nnz"])
    if op in ("update", "step"):
        F.update_device(s["val2"].data_ptr(), s["nnz"], s["mod"])
    if s["host"]:
        return F.Solve(s["b"])
    if op == "apply":
        F.apply_device(s["b"].data_ptr(), s["x"].data_ptr(), nrhs, n)
    else:
        F.solve_device(s["b"].data_ptr(), s["x"].data_ptr(), nrhs, n)
    return s["x"]


def _fronts(dim, N, width, leaf):
    s = mfgpu.Symbolic(dim, N, width, leaf)
    f = [s.front(i) for i in range(s.n_fronts)]
    return s, np.array([x["n"] for x in f], float), np.array([x["m"] for x in f], float)


def work(case):
    """Cholesky-form factorization flops n^3/3 + n^2 m + n m^2 per front (LU:
    twice), 2 (n^2 + 2 n m) per front and right-hand side of a solve; bytes:
    matrix values in, L written by a factorization, L read once by a solve, the
    vectors in and out."""
    op, nrhs = case["op"], case["nrhs"]
    esz = 4 if case["precision"] == "mixed" else 8
    if op == "batch":
        probs = [(2, (m, m), 1, case["leaf"]) for m in _sides(case)]
    else:
        N = _grid(case)
        probs = [(len(N), N, case["width"], case["leaf"])]
    flops = bytes_ = 0.0
    for dim, N, width, leaf in probs:
        s, n, m = _fronts(dim, N, width, leaf)
        lu = 2 if width > 1 else 1
        each = (n ** 3 / 3 + n ** 2 * m + n * m ** 2) * lu
        panel = (n * (n + 1) / 2 + n * m) * lu
        ndof = math.prod(N)
        values = ndof * (2 * dim * width + 1) * 8
        flops += float((2 * (n * n + 2 * n * m)).sum()) * nrhs
        bytes_ += float(panel.sum()) * esz + 2 * 8 * ndof * nrhs
        if op in ("factor", "step", "batch"):
            flops += float(each.sum())
            bytes_ += values + float(panel.sum()) * esz
        if op in ("update", "step"):
            lo, side = _patch(case)
            box = np.meshgrid(*[np.arange(max(0, l - 1), min(k, l + side + 1))
                                for l, k in zip(lo, N)], indexing="ij")
            strides = [math.prod(N[:d]) for d in range(dim)]
            dirty, _ = s.dirty(sum(g.ravel() * st for g, st in zip(box, strides)))
            flops += float(each[dirty].sum())
            bytes_ += values + float(panel[dirty].sum()) * esz
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------
# the exact result: the stencil on grid arrays, in plain numpy and torch
# ---------------------------------------------------------------------------
class _Operator:
    """-div(a grad u) on the grid, arrays indexed (z,) y, x.  `off` holds, per
    axis and distance, the weights of the neighbours below and above."""

    C = {1: [0.0, -1.0], 2: [0.0, -4 / 3, 1 / 12], 3: [0.0, -3 / 2, 3 / 20, -1 / 90]}

    def __init__(self, a, w):
        a = a.T                                     # x fastest
        dim, c = a.ndim, self.C[w]
        self.dim, self.w, self.shape = dim, w, [k - 2 * w for k in a.shape]

        def at(axis, k):
            return a[tuple(slice(w + (k if d == axis else 0), w + (k if d == axis else 0) + m)
                           for d, m in enumerate(self.shape))]

        diag, self.off = np.zeros(self.shape), []
        for k in range(w, 0, -1):
            for axis in range(dim - 1, -1, -1):     # x, y, (z)
                lo, up = 0.5 * (at(axis, -k) + at(axis, 1 - k)), 0.5 * (at(axis, k) + at(axis, k - 1))
                diag = diag - c[k] * (lo + up)
                self.off.append((axis, k, c[k] * lo, c[k] * up))
        self.diag = diag

    def parts(self, conv):
        """Diagonal and neighbour weights, each converted by `conv`."""
        return conv(self.diag), [(x, k, conv(l), conv(u)) for x, k, l, u in self.off]

    def product(self, u, parts):
        """A u for u of shape (nrhs, *grid)."""
        diag, off = parts
        y = diag * u
        for axis, k, lo, up in off:
            head = (slice(None),) * axis
            f, t = head + (slice(None, -k),), head + (slice(k, None),)
            b = (slice(None),)
            y[b + t] += lo[t] * u[b + f]
            y[b + f] += up[f] * u[b + t]
        return y


def _cg(op, parts, b, tol):
    """Conjugate gradients with diagonal scaling, every right-hand side at once."""
    axes = tuple(range(1, b.ndim))

    def dot(u, v):
        return (u * v).sum(axes, keepdim=True)

    x, r = torch.zeros_like(b), b.clone()
    z = r / parts[0]
    p, rz = z.clone(), dot(r, z)
    stop = dot(b, b) * tol * tol
    for it in range(40000):
        q = op.product(p, parts)
        alpha = rz / dot(p, q)
        x += alpha * p
        r -= alpha * q
        if it % 50 == 49 and bool((dot(r, r) <= stop).all()):
            break
        z = r / parts[0]
        new = dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return x


def _dense_solver(op, parts):
    """LU of the matrix as a dense array (the wider, nonsymmetric stencils)."""
    n = math.prod(op.shape)
    ids = torch.arange(n, device=parts[0].device).reshape(op.shape)
    A = torch.zeros((n, n), dtype=torch.float64, device=parts[0].device)
    A[ids.ravel(), ids.ravel()] = parts[0].ravel()
    for axis, k, lo, up in parts[1]:
        head = (slice(None),) * axis
        f, t = head + (slice(None, -k),), head + (slice(k, None),)
        A[ids[t].ravel(), ids[f].ravel()] = lo[t].ravel()
        A[ids[f].ravel(), ids[t].ravel()] = up[f].ravel()
    lu = torch.linalg.lu_factor(A)
    return lambda r, tol: torch.linalg.lu_solve(*lu, r.reshape(len(r), n).T).T.reshape(r.shape)


def _solution(a, w, b):
    """A^{-1} b for b (nrhs, n): FP64 solves, residuals in extended precision."""
    op = _Operator(a, w)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    parts = op.parts(lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev))
    wide = op.parts(lambda v: v.astype(np.longdouble))
    inner = _dense_solver(op, parts) if w > 1 else lambda r, tol: _cg(op, parts, r, tol)
    b = b.reshape(len(b), *op.shape).astype(np.longdouble)
    x, r = np.zeros_like(b), b
    for tol in (1e-8, 1e-6, 1e-4):
        size = np.abs(r).max()
        if size == 0:
            break
        d = inner(torch.from_numpy((r / size).astype(np.float64)).to(dev), tol)
        x = x + d.cpu().numpy().astype(np.longdouble) * size
        r = b - op.product(x, wide)
    return x.reshape(len(b), -1).astype(np.float64)


def exact(case, seed):
    if case["op"] == "batch":
        sides = _sides(case)
        b = _rhs(case, sum(m * m for m in sides), seed)
        out, at = [], 0
        for i, m in enumerate(sides):
            out.append(_solution(_coefficients(case, (m, m), seed * 1000 + i), 1,
                                 b[:, at:at + m * m]))
            at += m * m
        return np.concatenate(out, axis=1)
    N = _grid(case)
    a = _coefficients(case, N, seed)
    b = _rhs(case, math.prod(N), seed)
    if case["op"] in ("update", "step"):
        a = _changed(case, a)
    if case["op"] == "apply":
        op = _Operator(a, case["width"])
        y = op.product(b.reshape(len(b), *op.shape).astype(np.longdouble),
                       op.parts(lambda v: v.astype(np.longdouble)))
        return y.reshape(len(b), -1).astype(np.float64)
    x = _solution(a, case["width"], b)
    return x.T if case["host"] else x
