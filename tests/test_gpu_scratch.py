"""GPU: what a handle reserves.  The scratch and the tables of kernels that only
a switch or the autotuner reaches are made for those alone, and are there when
they are: in handles, in serving views and after an autotuning factorization."""
import numpy as np
import pytest
import torch

from mfgpu import MF2D, MFGPU_FP64, MFGPU_MIXED, Server, Symbolic, stencil
from problems import patch_update, problem, rel

pytestmark = pytest.mark.gpu

N = (63, 63)


@pytest.mark.parametrize("precision", [MFGPU_FP64, MFGPU_MIXED])
def test_a_small_handle_holds_little_device_memory(precision):
    _, A, b = problem(2, N, seed=81)
    warm = MF2D(A, *N, 1, 4, precision=precision)      # the library's own set-up
    warm.Factor()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    F = MF2D(A, *N, 1, 4, precision=precision)
    torch.cuda.synchronize()
    held = free0 - torch.cuda.mem_get_info()[0]
    inf = F.info()
    assert held <= 4 * (inf["front_bytes"] + inf["sep_bytes"]) + (16 << 20), held


def test_served_request_with_panel_kernels(monkeypatch):
    a, A, b = problem(2, N, seed=82)
    monkeypatch.setenv("MFGPU_PANEL_MAX_N", "4096")
    F = MF2D(A, *N, 1, 4)
    F.Factor()
    S = Server(F, a, slots=2, pool_gb=0.5)
    tickets = [S.submit([20, 30], [29, 39], f, b[0]) for f in (0.5, 3.0)]
    for f, t in zip((0.5, 3.0), tickets):
        G = MF2D(stencil.build_laplacian(stencil.scale_box(a, [20, 30], 9, f)), *N, 1, 4)
        G.Factor()
        assert rel(S.wait(t)[0], G.Solve(b[0])) < 1e-12
    S.close()


def test_autotune_again_between_factorizations_and_updates():
    a, A, b = problem(2, (127, 127), seed=83)
    a2, _ = patch_update(a, (127, 127), 9, 10.0, seed=11)
    A2 = stencil.build_laplacian(a2)
    mod = stencil.modified_dofs(A, A2)
    ref = MF2D(A, 127, 127, 1, 4)
    ref.Factor()
    x = ref.Solve(b[0])
    ref.Update(A2, mod)
    x2 = ref.Solve(b[0])
    F = MF2D(A, 127, 127, 1, 4)
    for _ in range(2):
        F.Factor()
        F.Factor()                             # (the second run is captured as a graph)
        assert rel(F.Solve(b[0]), x) < 1e-12
        F.autotune(1)
        assert rel(F.Solve(b[0]), x) < 1e-12
        F.Update(A2, mod)
        assert rel(F.Solve(b[0]), x2) < 1e-12
        F.Update(A, mod)
        assert rel(F.Solve(b[0]), x) < 1e-12


def test_a_solve_reserves_its_vectors_and_workspace_only():
    """One right-hand side, FP64: the front workspace (2 N per front) and one
    vector; the second vector is the LU fronts' apply alone."""
    size = (511, 511)
    _, A, b = problem(2, size, seed=84)
    F = MF2D(A, *size, 1, 8)
    F.Factor()
    F.Solve(b[0])
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    F.Solve(np.ascontiguousarray(np.tile(b, (16, 1)).T))
    torch.cuda.synchronize()
    held = free0 - torch.cuda.mem_get_info()[0]
    sym = Symbolic(2, size, 1, 8)
    work = sum(2 * (f["n"] + f["m"]) for f in map(sym.front, range(sym.n_fronts)))
    # 16 right-hand sides in place of one: 15 more of each, and the allocator's
    # 2 MiB granules; a second vector would add 15 n doubles, 31 MB
    assert held <= 8 * 15 * (work + A.n) + (8 << 20), (held, 8 * 15 * work, 8 * 15 * A.n)
