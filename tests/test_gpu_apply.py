"""GPU: the factored operator applied to vectors (Apply) on grids whose fronts
end inside the kernels' 64-wide items and whose last leaf boxes are much larger
than the rest, for every right-hand-side class (1, up to 4, 8, 16, more than a
chunk), against the matrix itself.

Tolerance: A = L L^T holds to about N_front * eps of ||A||, and a product sums
at most a front's columns again: 1e-12 (FP64, fronts of a few hundred, eps
1.1e-16) and 1e-4 (the FP32 factor, eps 6e-8) of ||A x||, with a margin of ten
for the operator's conditioning on random vectors."""
import numpy as np
import pytest

from mfgpu import MF2D, MF3D, MFGPU_FP64, MFGPU_MIXED
from problems import problem, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [(11, 10), (31, 33), (77, 39), (130, 70), (13, 17, 11), (28, 21, 23)])
@pytest.mark.parametrize("nrhs", [1, 3, 6, 16, 19])
@pytest.mark.parametrize("precision,tol", [(MFGPU_FP64, 1e-12), (MFGPU_MIXED, 1e-4)])
def test_apply_matches_the_matrix(N, nrhs, precision, tol):
    _, A, b = problem(len(N), N, seed=3, nrhs=nrhs)
    F = (MF2D if len(N) == 2 else MF3D)(A, *N, 1, 4, precision=precision)
    F.Factor()
    y = F.Apply(b.T)
    ref = A.to_scipy() @ b.T
    for c in range(nrhs):
        assert rel(y[:, c], ref[:, c]) < tol


def test_apply_keeps_infinities_to_the_rows_that_read_them():
    """An infinite entry reaches only the rows whose fronts share its DOF's root path."""
    N = (63, 63)
    _, A, b = problem(2, N, seed=4)
    F = MF2D(A, *N, 1, 4)
    F.Factor()
    x = b[0].copy()
    x[0] = np.inf                       # a corner cell: eliminated in the first leaf
    y = F.Apply(x)
    far = np.array([i + j * 63 for j in range(40, 62) for i in range(40, 62)])
    ok = np.isfinite(y[far])
    ref = F.Apply(b[0])
    assert ok.any() and np.allclose(y[far][ok], ref[far][ok], rtol=1e-9, atol=1e-9)
