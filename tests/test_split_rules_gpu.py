"""FAST order without a preconditioner at 5 to 8 rows per thread: one, two and four threads per order thread, as the
number of systems decides, on both sides of every change, bit for bit against the oracle."""
import numpy as np
import pytest

import bilu
import helpers as H
from test_patterns_gpu import TOL, TRIANGULAR, batch, band, grid2d

pytestmark = pytest.mark.gpu
PATTERNS = {"tri_150": band(150, (-1, 1)), "tri_256": band(256, (-1, 1)), "penta_300": band(300, (-2, -1, 1, 2)),
            "triangular_22x23": grid2d(22, 23, TRIANGULAR), "tri_700": band(700, (-1, 1)),
            "triangular_31x31": grid2d(31, 31, TRIANGULAR), "tri_1024": band(1024, (-1, 1))}


@pytest.mark.parametrize("name", list(PATTERNS))
@pytest.mark.parametrize("nsys", [1, 152, 153, 305, 457, 609, 1000, 1500, 2500])
@pytest.mark.parametrize("staging", [-1, 16, 25])
def test_without_preconditioner(cuda, name, nsys, staging):
    rp, ci = PATTERNS[name]
    v, b = batch(rp, ci, 2, 12)
    r = -(-nsys // 2)
    g = H.gpu_solve(cuda, rp, ci, np.tile(v, (r, 1))[:nsys], np.tile(b, (r, 1))[:nsys], precond=bilu.PRECOND_NONE,
                    reduction=bilu.REDUCE_FAST, smem_staging=staging, **TOL)
    nt = g["info"]["threads"]
    assert g["info"]["solver_kernel"] == 1 and 4 * nt < len(rp) - 1 <= 8 * nt
    o = H.oracle_fast(rp, ci, v, b, bilu.PRECOND_NONE, nt, False, **TOL)
    for f in ("iters", "conv", "status", "res", "x", "true_res"):
        H.assert_bitwise(g[f][:2], o[f][:nsys], f"{name}: {f}")
        H.assert_bitwise(g[f][-1], o[f][(nsys - 1) % 2], f"{name}: {f}, last system")
