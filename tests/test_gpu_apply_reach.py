"""GPU: an entry of x that is not finite reaches the DOFs of the fronts that hold
its DOF, by the symbolic tree, and no others: every other row of the applied
operator is finite and that of the matrix."""
import numpy as np
import pytest

from mfgpu import MF2D, MF3D, Symbolic
from problems import problem, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [(63, 47), (77, 39), (13, 17, 11)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("nrhs", [1, 3, 16])
def test_apply_spreads_an_infinity_no_further_than_its_fronts(N, bad, nrhs):
    _, A, b = problem(len(N), N, seed=5, nrhs=nrhs)
    F = (MF2D if len(N) == 2 else MF3D)(A, *N, 1, 4)
    F.Factor()
    sym = Symbolic(len(N), N, 1, 4)
    dofs = [sym.front(f)["dofs"] for f in range(sym.n_fronts)]
    full = A.to_scipy() @ b.T
    for d in (0, A.n // 2, A.n - 1):
        reach = np.zeros(A.n, bool)
        for f in dofs:
            if (f == d).any():
                reach[f] = True
        assert 0 < reach.sum() < A.n
        x = b.T.copy()
        x[d, nrhs // 2] = bad
        y = F.Apply(x)
        for c in range(nrhs):
            rows = ~reach if c == nrhs // 2 else np.ones(A.n, bool)
            assert np.isfinite(y[rows, c]).all()
            assert rel(y[rows, c], full[rows, c]) < 1e-12
