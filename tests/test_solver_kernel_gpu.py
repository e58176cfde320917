"""bilu_plan_solver_kernel names the kernel a batch runs on, for every kernel of the library; and the reference-order ISAI
solver's two kernels, told apart by that name, give the same bits."""
import numpy as np
import pytest

import bilu
import helpers as H
from test_patterns_gpu import NINE, band, grid2d

pytestmark = pytest.mark.gpu
FAST = dict(reduction=bilu.REDUCE_FAST)
ISAI, PAR, ILU, NONE = bilu.PRECOND_ILU0_ISAI, bilu.PRECOND_PARILU0, bilu.PRECOND_ILU0, bilu.PRECOND_NONE
GRID16, GRID36, NINE16 = bilu.gen_stencil(1, 16, 16, 1, 1, 1)[:2], bilu.gen_stencil(1, 36, 36, 1, 1, 1)[:2], grid2d(16, 16, NINE)


@pytest.mark.parametrize("pattern,opts,nsys,name", [
    (GRID16, dict(precond=ISAI), 5, "k_bicgstab_isai_ref"),
    (GRID16, dict(precond=ISAI, threads_per_system=128), 5, "k_bicgstab"),
    (GRID16, dict(precond=ILU), 5, "k_bicgstab_rr_lu"),
    (NINE16, dict(precond=ILU), 5, "k_bicgstab_rr"),
    (GRID16, dict(precond=ILU, **FAST), 5, "k_bicgstab_rr_lu"),
    (GRID16, dict(precond=ILU, threads_per_system=128, smem_staging=16, **FAST), 5, "k_bicgstab_rr_occ"),
    (GRID16, dict(precond=ISAI, threads_per_system=128, **FAST), 5, "k_bicgstab_rr"),
    (GRID16, dict(precond=ISAI, **FAST), 5, "k_bicgstab_rr_split"),
    (GRID16, dict(precond=NONE, **FAST), 1500, "k_bicgstab_rr"),
    (GRID36, dict(precond=PAR), 5, "k_bicgstab_rr_wide"),
    (GRID36, dict(precond=NONE), 5, "k_bicgstab"),
    (GRID36, dict(precond=NONE), 1000, "k_bicgstab_rr_wide"),
    (GRID36, dict(precond=ISAI), 5, "k_bicgstab"),
    (band(1100, (-1, 1)), dict(precond=ILU, **FAST), 5, "k_bicgstab_rr_wide"),
])
def test_names(cuda, pattern, opts, nsys, name):
    with bilu.Plan(*pattern, **opts) as plan:
        assert plan.solver_kernel(nsys) == name


@pytest.mark.parametrize("precond", [ISAI, bilu.PRECOND_PARILU0_ISAI])
@pytest.mark.parametrize("fp32", [False, True])
def test_reference_isai_kernels_agree(cuda, precond, fp32):
    rp, ci, v, b = bilu.gen_stencil(1, 19, 13, 1, 700, seed=4)
    kw = dict(precond=precond, ilu_approach=3, factor_precision=bilu.FP32 if fp32 else bilu.FP64,
              tol_mode=bilu.TOL_REL, tol=1e-10)
    g, s = (H.gpu_solve(cuda, rp, ci, v, b, threads_per_system=t, **kw) for t in (0, 256))
    for f in ("iters", "conv", "status", "res", "x", "true_res"):
        H.assert_bitwise(g[f], s[f], f)
    assert np.all(g["conv"] == 1)
