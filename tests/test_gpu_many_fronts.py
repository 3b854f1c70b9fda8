"""GPU: levels of more than 8,192 fronts larger than 128 rows.

A batch of 40 problems of 255 x 255 (maxSideLength 8) has a leaf level of 10,240
fronts of up to 285 rows.  Its factorization, a localized update and the solves must
agree with handles of the problems alone (FP64: within 1e-12; mixed: every
problem at relative residual 2e-10, refinement to 1e-10), and FP64 must not fall
back to one launch per 32-column step and kernel.
"""
import numpy as np
import pytest

from mfgpu import MF2D, MFBatch, MFGPU_FP64, MFGPU_MIXED, Symbolic, stencil
from problems import patch_update, problem, rel

pytestmark = pytest.mark.gpu

COUNT, N, LEAF = 40, (255, 255), 8


def test_the_batch_has_such_a_level(lib):
    sym = Symbolic(0, None, batch=[(2, N, 1, LEAF)] * 2)
    fr = [sym.front(f) for f in range(sym.n_fronts)]
    leaf = [f["n"] + f["m"] for f in fr if f["level"] == sym.levels - 1]
    assert len(leaf) * COUNT // 2 > 8192 and max(leaf) > 128


@pytest.mark.parametrize("precision", [MFGPU_FP64, MFGPU_MIXED])
def test_large_level_factors_updates_and_solves(precision):
    mats, coef, rhs = [], [], []
    for p in range(COUNT):
        a, A, b = problem(2, N, seed=400 + p)
        coef.append(a)
        mats.append(A)
        rhs.append(b[0])
    B = MFBatch([(A, N, 1, LEAF) for A in mats], precision=precision)
    B.profile(True)
    B.Factor()
    prof = B.profile_read()
    assert prof["potrf"]["launches"] == 0          # a launch per 32-column step and kernel
    B.profile(False)

    def check(mats):
        X = B.split(B.Solve(B.join(rhs)))
        for p in range(COUNT):
            res = np.linalg.norm(mats[p].matvec(X[p][:, 0]) - rhs[p]) / np.linalg.norm(rhs[p])
            assert res <= (1e-12 if precision == MFGPU_FP64 else 2e-10)
        if precision == MFGPU_FP64:
            for p in (0, 17, COUNT - 1):
                F = MF2D(mats[p], *N, 1, LEAF)
                F.Factor()
                assert rel(X[p][:, 0], F.Solve(rhs[p])) < 1e-12
                F.close()
        return X

    before = check(mats)
    j = 17
    a2, _ = patch_update(coef[j], N, 9, 10.0, seed=6)
    A2 = stencil.build_laplacian(a2)
    B.Update([A2 if p == j else None for p in range(COUNT)],
             [stencil.modified_dofs(mats[j], A2) if p == j else [] for p in range(COUNT)])
    after = check(mats[:j] + [A2] + mats[j + 1:])
    assert rel(after[j], before[j]) > 1e-6
