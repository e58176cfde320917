"""FAST order at 5 to 8 rows per thread without ILU factors, where several
threads share an order thread's rows: every row count per thread, one warp to
four, few systems (four threads per order thread) and more than are resident at
once (two, or four on one warp), bit for bit against the oracle."""
import numpy as np
import pytest

import bilu
import helpers as H

pytestmark = pytest.mark.gpu
TOL = dict(tol_mode=bilu.TOL_REL, tol=1e-10)
GRIDS = [(9, 15, 1), (14, 13, 1), (16, 16, 1), (17, 16, 1), (8, 8, 6), (22, 22, 1), (20, 26, 1), (24, 24, 1),
         (11, 9, 6), (26, 30, 1), (10, 10, 10), (32, 32, 1)]


@pytest.mark.parametrize("grid", GRIDS, ids=["x".join(map(str, g)) for g in GRIDS])
@pytest.mark.parametrize("precond,fp32", [(bilu.PRECOND_ILU0_ISAI, True), (bilu.PRECOND_ILU0_ISAI, False),
                                          (bilu.PRECOND_NONE, False), (bilu.PRECOND_GENERAL_ISAI, True)])
@pytest.mark.parametrize("nsys", [3, 1300])
def test_split_rows_bitwise(cuda, grid, precond, fp32, nsys):
    kind = 2 if grid[2] > 1 else 1
    rp, ci, v, b = bilu.gen_stencil(kind, *grid, nsys, seed=sum(grid))
    kw = dict(isai_power=1) if precond == bilu.PRECOND_GENERAL_ISAI else {}
    g = H.gpu_solve(cuda, rp, ci, v, b, precond=precond, ilu_approach=3, reduction=bilu.REDUCE_FAST,
                    factor_precision=bilu.FP32 if fp32 else bilu.FP64, max_iter=40, **kw, **TOL)
    nt = g["info"]["threads"]
    assert g["info"]["solver_kernel"] == 1 and 4 * nt < len(rp) - 1 <= 8 * nt
    s = np.unique(np.linspace(0, nsys - 1, 3).astype(int))
    o = H.oracle_fast(rp, ci, v[s], b[s], precond, nt, fp32, approach=3, power=kw.get("isai_power", 2), max_iter=40,
                      **TOL)
    for f in ("iters", "conv", "status", "res", "x", "true_res"):
        H.assert_bitwise(g[f][s], o[f], f"{grid} precond {precond} fp32={fp32} nsys={nsys}: {f}")
