"""Reference-order solves whose three values per diagonal cost a resident CTA: batches around the sizes at which the
kernel with one value per diagonal takes over, 5 to 8 rows per thread, compact and general programs, bit for bit
against the oracle."""
import numpy as np
import pytest

import bilu
import helpers as H
from test_patterns_gpu import NINE, TOL, batch, band, grid2d

pytestmark = pytest.mark.gpu
FIELDS = ("iters", "conv", "status", "res", "x", "true_res")
PATTERNS = {"nine_28x28": grid2d(28, 28, NINE), "nine_22x23": grid2d(22, 23, NINE), "penta_256": band(256, (-2, -1, 1, 2)),
            "seven_point_10x10x10": bilu.gen_stencil(2, 10, 10, 10, 1, seed=1)[:2],
            "band_180": band(180, (-7, -5, -3, -1, 1, 2, 4, 6))}


@pytest.mark.parametrize("name", list(PATTERNS))
@pytest.mark.parametrize("precond", [bilu.PRECOND_ILU0, bilu.PRECOND_PARILU0])
@pytest.mark.parametrize("nsys", [3, 460, 1750, 2000])
def test_values_per_diagonal(cuda, name, precond, nsys):
    rp, ci = PATTERNS[name]
    v, b = batch(rp, ci, 2, 11)
    v[1, 0] = v[1, -1] = 0.0  # a zero pivot: the quotients' way out
    r = -(-nsys // 2)
    g = H.gpu_solve(cuda, rp, ci, np.tile(v, (r, 1))[:nsys], np.tile(b, (r, 1))[:nsys], precond=precond, **TOL)
    assert g["info"]["solver_kernel"] == 1
    o = H.oracle_pipeline(rp, ci, v, b, precond, **TOL)
    last = [(nsys - 2) % 2, (nsys - 1) % 2]
    for f in FIELDS:
        H.assert_bitwise(g[f][:2], o[f], f"{name}: {f}")
        H.assert_bitwise(g[f][-2:], o[f][last], f"{name}: {f}, last systems")
