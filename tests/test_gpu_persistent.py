"""The persistent BiCGStab (gpu_persistent, default 1): PBiCGStab and
MergedPBiCGStab with no preconditioner or a Jacobi preconditioner run every
iteration, the convergence test and the final update in one cooperative
launch with bounded grid barriers. It must give the iteration-by-iteration
path's results bit for bit (iterations, convergence flags, residuals,
solution), whether the solve converges or stops at max_iters, and a grid
barrier that can never complete must end in a reported timeout with the GPU
context still usable."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_solve import gpu_solve, true_rel_res

pytestmark = pytest.mark.gpu


def params(method, prec, persistent, max_iters=1000, sweeps=None, tol=1e-8):
    p = {"solver": {"method": method, "max_iters": max_iters, "rel_tolerance": tol,
                    "abs_tolerance": 0, "gpu_persistent": persistent}}
    if prec:
        p["preconditioner"] = {"method": "Jacobi"}
        if sweeps:
            p["preconditioner"]["max_iters"] = sweeps
    return p


@pytest.mark.parametrize("method,prec,nv,sweeps,grid,cap",
                         [("MergedPBiCGStab", True, 1, None, (32, 32, 32), 1000),
                          ("MergedPBiCGStab", True, 2, 3, (20, 19, 18), 1000),
                          ("PBiCGStab", True, 8, 1, (16, 16, 16), 1000),
                          ("PBiCGStab", False, 4, None, (17, 16, 15), 1000),
                          ("MergedPBiCGStab", True, 1, None, (32, 32, 32), 7)])
@pytest.mark.parametrize("share", [1, 3, 4])
def test_persistent_equals_stepwise(gpu, method, prec, nv, sweeps, grid, cap, share):
    """share (gpu_persistent): canonical blocks each block of the launch plays;
    the reductions stay per canonical block, so every share gives the same
    bits as the step-by-step solve."""
    row, col, val = gpu.generate_cube(*grid)
    n = len(row) - 1
    b = np.random.default_rng(nv + grid[0]).uniform(-1, 1, n * nv)
    out = {}
    for persistent in (0, share):
        k0 = gpu.kernel_launches()
        x, st, S = gpu_solve(gpu, row, col, val, nv, params(method, prec, persistent, cap, sweeps),
                             b)
        out[persistent] = (x, st, gpu.kernel_launches() - k0)
    (x0, s0, l0), (x1, s1, l1) = out[0], out[share]
    assert s0["iters"] == s1["iters"]
    assert s0["conv"].tolist() == s1["conv"].tolist()
    assert s0["rel_res"].tobytes() == s1["rel_res"].tobytes()
    assert s0["abs_res"].tobytes() == s1["abs_res"].tobytes()
    assert x0.tobytes() == x1.tobytes()
    assert l1 < l0 and l1 <= 3  # start, the persistent launch (a converged solve: no more)
    if cap < 1000:
        assert s1["iters"] == cap and not s1["conv"].any()
    else:
        assert s1["conv"].all()
        assert true_rel_res(row, col, val, x1, b, nv).max() <= 1e-7


@pytest.mark.parametrize("stencil,nv,grid,sweeps", [(27, 1, (32, 31, 33), None),
                                                    (7, 16, (15, 14, 11), 1), (7, 32, (11, 10, 9), 2),
                                                    (7, 8, (17, 16, 15), 4), (7, 8, (17, 16, 15), 5),
                                                    (7, 4, (40, 39, 38), None)])
def test_persistent_forms(gpu, stencil, nv, grid, sweeps):
    """The register-resident form at its edges (nearly one block an SM, all lanes
    of a warp on one row, long rows, as many Jacobi sweeps as it takes) and what
    is beyond it (one sweep more, a larger system): the bits of the step-by-step
    solve."""
    row, col, val = gpu.generate_diffusion(stencil, *grid, 1.0, 1.0, 4)
    n = len(row) - 1
    b = np.random.default_rng(nv).uniform(-1, 1, n * nv)
    x0, s0, _ = gpu_solve(gpu, row, col, val, nv,
                          params("MergedPBiCGStab", True, 0, sweeps=sweeps), b)
    x1, s1, _ = gpu_solve(gpu, row, col, val, nv,
                          params("MergedPBiCGStab", True, 1, sweeps=sweeps), b)
    assert s0["iters"] == s1["iters"] and s1["conv"].all()
    assert s0["rel_res"].tobytes() == s1["rel_res"].tobytes()
    assert x0.tobytes() == x1.tobytes()
    # another right-hand side on the same solver: nothing is left of the first solve
    M, X, B = matrix_and_vectors(gpu, row, col, val, nv)
    S2 = gpu.Solver(M, gpu.Params(params("MergedPBiCGStab", True, 1, sweeps=sweeps)), X, B)
    for rhs in (b[::-1].copy(), b):
        B.upload(rhs)
        X.set(0.0)
        S2.solve()
    assert X.download().tobytes() == x0.tobytes()


def matrix_and_vectors(gpu, row, col, val, nv):
    M = gpu.Matrix(row, col, val)
    return M, gpu.Vector(M.n, nv, M.part), gpu.Vector(M.n, nv, M.part)


def test_grid_barrier_wait_runs_out(gpu):
    t = C.c_int(-1)
    gpu.call("XAMG_b200_grid_selftest", 0.05, C.byref(t))
    assert t.value == 1
    # the context is still usable: a persistent solve right after
    row, col, val = gpu.generate_cube(12, 12, 12)
    b = np.ones(len(row) - 1)
    x, st, S = gpu_solve(gpu, row, col, val, 1, params("MergedPBiCGStab", True, 1), b)
    assert st["conv"].all()


@pytest.mark.parametrize("stencil,nv,edge,one_launch", [(7, 2, 39, True), (27, 2, 39, False),
                                                        (7, 2, 45, False), (27, 2, 36, True),
                                                        (7, 4, 33, False), (7, 16, 18, False)])
def test_systems_past_three_blocks_an_sm(gpu, stencil, nv, edge, one_launch):
    """More canonical blocks than three an SM: one launch takes them on short rows at
    nv = 2, the separate launches otherwise; the same bits either way."""
    row, col, val = gpu.generate_diffusion(stencil, edge, edge, edge, 1.0, 1.0, 4)
    n = len(row) - 1
    b = np.random.default_rng(nv).uniform(-1, 1, n * nv)
    x0, s0, _ = gpu_solve(gpu, row, col, val, nv, params("MergedPBiCGStab", True, 0), b)
    k0 = gpu.kernel_launches()
    x1, s1, _ = gpu_solve(gpu, row, col, val, nv, params("MergedPBiCGStab", True, 1), b)
    assert (gpu.kernel_launches() - k0 < s1["iters"]) == one_launch
    assert s0["iters"] == s1["iters"] and s1["conv"].all()
    assert x0.tobytes() == x1.tobytes()
