"""GPU: the forward / backward sweeps on grids whose fronts end inside the
32-column blocks (and whose last leaf boxes are much larger than the rest), for
every right-hand-side class (1, up to 4, 8, 16, more than a chunk), Cholesky and
pivoted LU fronts, against a sparse direct solve of the same matrix.

Tolerances: FP64 1e-11 (condition number of these grids at contrast 100: below
1e5, times eps and the few hundred operations of a path through the tree);
mixed: the refinement's own target, 1e-10 in the residual, times the same
condition number over the norm ratio of a random right-hand side (1e-8)."""
import numpy as np
import pytest

from mfgpu import MF2D, MF3D, MFGPU_FP64, MFGPU_MIXED, stencil
from problems import SEED0, problem, rel

pytestmark = pytest.mark.gpu


def _solve(A, b):
    import scipy.sparse.linalg as sl
    lu = sl.splu(A.to_scipy().tocsc())
    return lu.solve(np.asfortranarray(b))


@pytest.mark.parametrize("N", [(10, 10), (31, 33), (77, 39), (130, 70), (13, 17, 11), (28, 21, 23)])
@pytest.mark.parametrize("nrhs", [1, 3, 6, 16, 19])
@pytest.mark.parametrize("precision,tol", [(MFGPU_FP64, 1e-11), (MFGPU_MIXED, 1e-8)])
def test_solve_matches_a_sparse_direct_solve(N, nrhs, precision, tol):
    _, A, b = problem(len(N), N, seed=5, nrhs=nrhs)
    F = (MF2D if len(N) == 2 else MF3D)(A, *N, 1, 4, precision=precision)
    F.Factor()
    x, ref = F.Solve(b.T), _solve(A, b.T)
    for c in range(nrhs):
        assert rel(x[:, c], ref[:, c]) < tol


@pytest.mark.parametrize("N", [(31, 33), (77, 39), (130, 70), (28, 21, 23), (31, 31, 31)])
@pytest.mark.parametrize("nrhs", [1, 3, 8, 9, 16, 19])
@pytest.mark.parametrize("precision,tol", [(MFGPU_FP64, 1e-11), (MFGPU_MIXED, 1e-8)])
def test_flag_ordered_sweeps_match_a_sparse_direct_solve(monkeypatch, N, nrhs, precision, tol):
    """The flag-ordered sweeps on every level with a front of 48 or more rows:
    block edges at 64, pivot and boundary rows in one block, fronts of one block."""
    monkeypatch.setenv("MFGPU_SOLVE_COOP_MIN_N", "48")
    _, A, b = problem(len(N), N, seed=8, nrhs=nrhs)
    F = (MF2D if len(N) == 2 else MF3D)(A, *N, 1, 4, precision=precision)
    F.Factor()
    x, ref = F.Solve(b.T), _solve(A, b.T)
    for c in range(nrhs):
        assert rel(x[:, c], ref[:, c]) < tol


@pytest.mark.parametrize("nrhs", [1, 5, 16])
@pytest.mark.parametrize("precision,tol", [(MFGPU_FP64, 1e-11), (MFGPU_MIXED, 1e-8)])
def test_large_fronts_of_a_level_of_many(monkeypatch, tmp_path, nrhs, precision, tol):
    """A leaf level of 1024 fronts whose last ones are several times larger: those
    go to the flag-ordered sweeps.  A factor saved under another split of the
    level loads and solves as well."""
    N = (270, 150)
    monkeypatch.setenv("MFGPU_SOLVE_COOP_MIN_N", "120")
    _, A, b = problem(2, N, seed=9, nrhs=nrhs)
    F = MF2D(A, *N, 1, 4, precision=precision)
    F.Factor()
    x, ref = F.Solve(b.T), _solve(A, b.T)
    for c in range(nrhs):
        assert rel(x[:, c], ref[:, c]) < tol
    F.save(tmp_path / "f")
    monkeypatch.setenv("MFGPU_SOLVE_COOP_MIN_N", "200")
    G = MF2D(A, *N, 1, 4, precision=precision)
    G.load(tmp_path / "f")
    y = G.Solve(b.T)
    for c in range(nrhs):
        assert rel(y[:, c], ref[:, c]) < tol


@pytest.mark.parametrize("N,width", [((31, 33), 2), ((77, 39), 2), ((50, 41), 3), ((13, 11, 12), 2)])
@pytest.mark.parametrize("nrhs", [1, 3, 6, 16])
def test_lu_solve_matches_a_sparse_direct_solve(N, width, nrhs):
    a = stencil.loguniform_coefficients(N, 0.5, 2.0, SEED0 + 6, width=width)
    A = stencil.build_laplacian(a, width=width)
    b = stencil.uniform_rhs(A.n, nrhs, SEED0 + 7)
    F = (MF2D if len(N) == 2 else MF3D)(A, *N, width, 4)
    F.Factor()
    x, ref = F.Solve(b.T), _solve(A, b.T)
    for c in range(nrhs):
        assert rel(x[:, c], ref[:, c]) < 1e-11
