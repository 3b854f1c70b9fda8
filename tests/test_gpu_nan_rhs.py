"""GPU, mixed precision: a right-hand side whose residual is not a number misses
the tolerance (MFGPU_ERR_NOT_CONVERGED, residual NaN); the other columns and the
other problems of a batch are solved and handed out all the same."""
import math

import numpy as np
import pytest
import torch

from mfgpu import MF2D, MFBatch, MFGPU_MIXED, MFError, _lib
from problems import problem

pytestmark = pytest.mark.gpu


def relres(A, x, b):
    return float(np.linalg.norm(A.matvec(x) - b) / np.linalg.norm(b))


def solve_device(F, b):
    """x of b (nrhs, n) through device buffers; the call's error status, or 0."""
    d = torch.from_numpy(b).cuda()
    x = torch.zeros_like(d)
    torch.cuda.synchronize()
    status = 0
    try:
        F.solve_device(d.data_ptr(), x.data_ptr(), b.shape[0], b.shape[1])
    except MFError as e:
        status = e.status
    torch.cuda.synchronize()
    return x.cpu().numpy(), status


@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("nrhs,col", [(1, 0), (3, 1), (18, 2)])
def test_a_column_that_is_not_a_number_is_reported(bad, nrhs, col):
    N = (63, 63)
    _, A, b = problem(2, N, seed=64, nrhs=nrhs)
    F = MF2D(A, *N, 1, 4, precision=MFGPU_MIXED)
    F.Factor()
    b[col, 100] = bad
    with pytest.raises(MFError) as ei:
        F.Solve(b.T)
    assert ei.value.status == _lib.MFGPU_ERR_NOT_CONVERGED
    assert math.isnan(F.stats()["residual"])
    x, status = solve_device(F, b)
    assert status == _lib.MFGPU_ERR_NOT_CONVERGED and math.isnan(F.stats()["residual"])
    for c in range(nrhs):
        if c != col:
            assert relres(A, x[c], b[c]) <= 2e-10
    good = np.delete(b, col, axis=0)
    if nrhs > 1:                                  # the handle stays usable
        x, status = solve_device(F, good)
        assert status == 0 and F.stats()["residual"] <= 1e-10


def test_a_member_that_is_not_a_number_leaves_the_others():
    sides = [31, 63, 40]
    probs = [problem(2, (m, m), seed=70 + m) for m in sides]
    B = MFBatch([(A, (m, m), 1, 4) for m, (_, A, _) in zip(sides, probs)], precision=MFGPU_MIXED)
    B.Factor()
    rhs = B.join([b[0] for _, _, b in probs])
    rhs[B.offsets[1] + 7] = math.nan
    x, status = solve_device(B, np.ascontiguousarray(rhs.T))
    assert status == _lib.MFGPU_ERR_NOT_CONVERGED
    xs = B.split(x.T)
    for p in (0, 2):
        assert relres(probs[p][1], xs[p][:, 0], probs[p][2][0]) <= 2e-10
