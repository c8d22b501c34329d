"""The block-wise Gauss-Seidel sweep (csrc/hsgs.cuh) against the oracle, bit for
bit, where its forms meet: Gauss-Seidel blocks of 8 to 40 rows and one block of
the whole level (swept from global memory when it does not fit in shared
memory), one to thirty-two lanes a warp, one to three sweeps from zero and
from a non-zero x, FP64 and FP32 levels, in-block columns of one and four bytes
(without narrowing the lagged term stays a kernel of its own)."""
import pytest

from test_gpu_solve import MG_BASE, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv,rows,sweeps,reduced,narrow",
                         [(1, 32, 1, 0, 1), (1, 8, 2, 1, 1), (1, 20000, 1, 0, 1),
                          (2, 32, 3, "full32", 2), (4, 8, 2, 0, 0), (8, 32, 2, "full32", 2),
                          (16, 30, 1, 1, 1), (32, 32, 2, 0, 1), (32, 300, 1, 0, 1)])
def test_hsgs_forms(gpu, oracle, nv, rows, sweeps, reduced, narrow):
    row, col, val = gpu.generate_diffusion(7, 19, 17, 13, 1.0, 1.0, 2)
    sm = {"method": "HSGS", "max_iters": sweeps, "gpu_hsgs_rows": rows}
    prec = dict(MG_BASE, method="MultiGrid", mg_reduced_precision=int(reduced == 1),
                gpu_index_compress=narrow)
    if reduced == "full32":
        prec["gpu_precond_f32"] = 1
    params = {"solver": {"method": "MergedPBiCGStab", "max_iters": 100, "rel_tolerance": 1e-8,
                         "abs_tolerance": 0, "gpu_index_compress": narrow},
              "preconditioner": prec, "pre_smoother": sm, "post_smoother": dict(sm),
              "coarse_grid_solver": {"method": "Direct"}}
    st, _ = check(gpu, oracle, row, col, val, nv, params, seed=nv + rows, hsgs_rows=rows)
    assert st["conv"].all()


@pytest.mark.parametrize("nv,off", [(8, (-2, False)), (1, (4, True))])
def test_off_block_columns(gpu, oracle, nv, off):
    """Two-byte relative columns (gpu_index_compress = 2) of a level of more than
    65,536 rows whose lagged term stays a SpMV; absolute ones where the sweep
    forms it."""
    row, col, val = gpu.generate_diffusion(7, 41, 41, 41, 1.0, 1.0, 3)
    sm = {"method": "HSGS", "max_iters": 1}
    params = {"solver": {"method": "MergedPBiCGStab", "max_iters": 100, "rel_tolerance": 1e-8,
                         "abs_tolerance": 0, "gpu_index_compress": 2},
              "preconditioner": dict(MG_BASE, method="MultiGrid", gpu_precond_f32=1,
                                     gpu_index_compress=2, mg_coarse_matrix_size=500),
              "pre_smoother": sm, "post_smoother": dict(sm),
              "coarse_grid_solver": {"method": "Direct"}}
    st, S = check(gpu, oracle, row, col, val, nv, params, seed=1)
    assert st["conv"].all()
    assert S.level_hsgs(0) == off
    # at most 65,536 columns on the coarser levels
    assert all(S.level_hsgs(lv)[0] in (1, 2) for lv in range(1, S.nlevels() - 1))
