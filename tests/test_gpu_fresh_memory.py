"""GPU: results do not depend on what freshly allocated device memory holds.
Handles whose sweep scratch starts as all ones (NaNs) are made, solved and closed
first, so that the next handles' small buffers may lie in what they gave back."""
import numpy as np
import pytest

from mfgpu import MF2D, MF3D, MFGPU_FP64, MFGPU_MIXED
from problems import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [(63, 63), (130, 70), (17, 16, 15)])
@pytest.mark.parametrize("precision", [MFGPU_FP64, MFGPU_MIXED])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_solve_and_apply_on_memory_given_back_full_of_nans(monkeypatch, N, precision, nrhs):
    _, A, b = problem(len(N), N, seed=12, nrhs=nrhs)
    make = MF2D if len(N) == 2 else MF3D
    for count in (16, 16, 1):
        monkeypatch.setenv("MFGPU_SOLVE_COOP_MIN_N", "16")
        held = [make(A, *N, 1, 4) for _ in range(8)]
        for H in held:
            H.Factor()
            H.Solve(np.tile(b[0][:, None], (1, count)))
        for H in held:
            H.close()
        monkeypatch.delenv("MFGPU_SOLVE_COOP_MIN_N")
        F = make(A, *N, 1, 4, precision=precision)
        F.Factor()
        for k in range(1, nrhs + 1):        # buffers that grow start afresh
            x = F.Solve(b[:k].T)
            assert np.isfinite(x).all() and np.isfinite(F.Apply(b[:k].T)).all()
            r = A.to_scipy() @ x - b[:k].T
            assert np.linalg.norm(r) / np.linalg.norm(b[:k]) < 1e-9
