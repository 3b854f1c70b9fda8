"""GPU: a factor file whose block inverses belong to another set of fronts of the
same total size (the set follows the sweeps' threshold) must not be taken as
this handle's: the loaded factor solves like the handle's own."""
import numpy as np
import pytest

from mfgpu import MF2D, MFGPU_MIXED
from problems import problem, rel

pytestmark = pytest.mark.gpu


def test_equal_sizes_of_different_sets_are_told_apart(monkeypatch, tmp_path):
    # thresholds 20 and 30 give both 508 blocks of 64 x 64, in other fronts
    N = (130, 280)
    _, A, b = problem(2, N, seed=63)
    monkeypatch.setenv("MFGPU_SOLVE_COOP_MIN_N", "20")
    F = MF2D(A, *N, 1, 3, precision=MFGPU_MIXED)
    F.Factor()
    F.save(tmp_path / "f")
    monkeypatch.setenv("MFGPU_SOLVE_COOP_MIN_N", "30")
    G = MF2D(A, *N, 1, 3, precision=MFGPU_MIXED)
    G.Factor()
    G.save(tmp_path / "g")
    assert (tmp_path / "f").stat().st_size == (tmp_path / "g").stat().st_size
    # refinement to 1e-10 takes as many steps as with the handle's own inverses
    x = G.Solve(b[0])
    steps = G.stats()["iterations"]
    G.load(tmp_path / "f")
    y = G.Solve(b[0])
    assert G.stats()["iterations"] <= steps + 1
    assert rel(y, x) < 1e-8
    assert np.linalg.norm(A.matvec(y) - b[0]) / np.linalg.norm(b[0]) <= 2e-10
