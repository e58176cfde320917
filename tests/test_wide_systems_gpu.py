"""Systems of 1025 to 2048 rows on the register-resident solver: in the
reference's order against the oracle, and in the FAST order (whose bits are
the shared-memory solver's) against that solver, which 1024 threads per system
still select."""
import numpy as np
import pytest

import bilu
import helpers as H

pytestmark = pytest.mark.gpu
FIELDS = ("iters", "conv", "status", "res", "x", "true_res")
GRIDS = [(41, 25, 1), (36, 36, 1), (48, 32, 1), (29, 53, 1), (64, 32, 1), (11, 10, 10)]
PRECONDS = [(bilu.PRECOND_ILU0, False), (bilu.PRECOND_ILU0_SPLIT, True), (bilu.PRECOND_PARILU0, False),
            (bilu.PRECOND_PARILU0, True), (bilu.PRECOND_NONE, False)]


def _batch(grid):
    kind = 2 if grid[2] > 1 else 1
    return bilu.gen_stencil(kind, *grid, 3, seed=sum(grid))


@pytest.mark.parametrize("grid", GRIDS, ids=["x".join(map(str, g)) for g in GRIDS])
@pytest.mark.parametrize("precond,fp32", PRECONDS)
def test_reference_order_bitwise(cuda, grid, precond, fp32):
    rp, ci, v, b = _batch(grid)
    kw = dict(tol_mode=bilu.TOL_REL, tol=1e-10, max_iter=60)
    o = H.oracle_pipeline(rp, ci, v, b, precond, fp32=fp32, **kw)
    g = H.gpu_solve(cuda, rp, ci, v, b, precond=precond, factor_precision=bilu.FP32 if fp32 else bilu.FP64, **kw)
    assert g["info"]["solver_kernel"] == 1
    for f in FIELDS:
        H.assert_bitwise(g[f], o[f], f"{grid} precond {precond} fp32={fp32}: {f}")


@pytest.mark.parametrize("grid", GRIDS, ids=["x".join(map(str, g)) for g in GRIDS])
@pytest.mark.parametrize("precond,fp32", PRECONDS)
def test_fast_order_keeps_its_bits(cuda, grid, precond, fp32):
    rp, ci, v, b = _batch(grid)
    kw = dict(tol_mode=bilu.TOL_REL, tol=1e-10, max_iter=60, precond=precond, reduction=bilu.REDUCE_FAST,
              factor_precision=bilu.FP32 if fp32 else bilu.FP64)
    g = H.gpu_solve(cuda, rp, ci, v, b, **kw)
    s = H.gpu_solve(cuda, rp, ci, v, b, threads_per_system=1024, **kw)
    assert g["info"]["solver_kernel"] == 1 and s["info"]["solver_kernel"] == 0
    for f in FIELDS:
        H.assert_bitwise(g[f], s[f], f"{grid} precond {precond} fp32={fp32}: {f}")


def test_tiny_and_zero_rhs_and_nan(cuda):
    rp, ci, v, b = _batch((36, 36, 1))
    b[0] = 0.0
    b[1] *= 1e-14
    v[2, 7] = np.nan
    o = H.oracle_pipeline(rp, ci, v, b, bilu.PRECOND_ILU0, max_iter=4)
    g = H.gpu_solve(cuda, rp, ci, v, b, precond=bilu.PRECOND_ILU0, max_iter=4)
    for f in FIELDS[:5]:
        H.assert_bitwise(g[f], o[f], f)
