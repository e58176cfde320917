"""The reference-order ISAI solver with several systems per CTA
(csrc/k_solve_isai_ref.cu) against the oracle, bit for bit: row trees of 2D, 3D
and general rows, one system per CTA and several (full and partly filled CTAs,
systems that stop at different iterations), FP64 and FP32 ISAI, edge cases."""
import numpy as np
import pytest

import bilu
import helpers as H
from test_parity_gpu import _random_pattern_batch

pytestmark = pytest.mark.gpu
FIELDS = ("iters", "conv", "status", "res", "x", "true_res")
GRIDS = [(6, 6, 1), (8, 8, 1), (13, 5, 1), (16, 16, 1), (17, 16, 1), (24, 24, 1), (32, 32, 1), (5, 5, 5), (7, 7, 7),
         (10, 10, 10)]


def _check(cuda, rp, ci, v, b, precond, sample, **kw):
    g = H.gpu_solve(cuda, rp, ci, v, b, precond=precond, ilu_approach=3, **kw)
    assert g["info"]["solver_kernel"] == 0
    okw = {k: kw[k] for k in ("tol_mode", "tol", "max_iter", "isai_power") if k in kw}
    o = H.oracle_pipeline(rp, ci, v[sample], b[sample], precond, approach=3,
                          fp32=kw.get("factor_precision", 0) == bilu.FP32, **okw)
    for f in FIELDS:
        H.assert_bitwise(g[f][sample], o[f], f"precond {precond} n={len(rp) - 1} nsys={len(b)}: {f}")
    return g


@pytest.mark.parametrize("grid", GRIDS, ids=["x".join(map(str, g)) for g in GRIDS])
@pytest.mark.parametrize("nsys", [1, 5, 1700])
@pytest.mark.parametrize("fp32", [False, True])
def test_several_systems_per_cta_bitwise(cuda, grid, nsys, fp32):
    rp, ci, v, b = bilu.gen_stencil(2 if grid[2] > 1 else 1, *grid, nsys, seed=nsys + sum(grid))
    kw = dict(tol_mode=bilu.TOL_REL, tol=1e-10, factor_precision=bilu.FP32) if fp32 else {}
    s = np.unique(np.concatenate([np.linspace(0, nsys - 1, 6), [nsys - 1, max(nsys - 2, 0)]]).astype(int))
    g = _check(cuda, rp, ci, v, b, bilu.PRECOND_ILU0_ISAI, s, **kw)
    assert np.all(g["conv"] == 1)


@pytest.mark.parametrize("precond", [bilu.PRECOND_ILU0_ISAI, bilu.PRECOND_PARILU0_ISAI])
def test_general_rows_bitwise(cuda, precond):
    rp, ci, v, b = _random_pattern_batch(640)
    _check(cuda, rp, ci, v, b, precond, np.arange(0, 640, 91), isai_power=1)


@pytest.mark.parametrize("max_iter", [0, 1, 2, 500])
def test_stopped_systems_beside_others(cuda, max_iter):
    """Systems that never start, stop early, break down or run on share a CTA."""
    rp, ci, v, b = H.workload("2d5_16x16", 2000)
    for s in range(0, 2000, 7):
        b[s] = 0.0
        b[s + 1] *= 1e-14
        v[s + 2, 3] = np.nan
        b[s + 3] *= 1e-6
    _check(cuda, rp, ci, v, b, bilu.PRECOND_ILU0_ISAI, np.arange(0, 30), max_iter=max_iter)
