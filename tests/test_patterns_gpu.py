"""Shared patterns that are not full stencils: triangles of at most three
entries per row with dependency pairs off the diagonals (triangular lattice,
pentadiagonal), stencils with couplings missing on one side, random patterns
with wide levels.  The factorisation and every ILU solver form against the
oracle, bit for bit."""
import numpy as np
import pytest

import bilu
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu
FIELDS = ("iters", "conv", "status", "res", "x", "true_res")
TOL = dict(tol_mode=bilu.TOL_REL, tol=1e-10, max_iter=40)
TRIANGULAR = [(0, 0), (1, 0), (-1, 0), (0, 1), (0, -1), (1, 1), (-1, -1)]
NINE = [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)]


def csr(rows):
    rows = [sorted(set(r)) for r in rows]
    return (np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32),
            np.concatenate([np.array(r, np.int32) for r in rows]))


def grid2d(gx, gy, offsets):
    return csr([[(y + b) * gx + x + a for a, b in offsets if 0 <= x + a < gx and 0 <= y + b < gy]
                for y in range(gy) for x in range(gx)])


def band(n, offsets):
    return csr([[i] + [i + o for o in offsets if 0 <= i + o < n] for i in range(n)])


def one_sided(gx, gy, gz, seed):
    """A stencil without a random share of its couplings, each direction by itself."""
    rp, ci, _, _ = bilu.gen_stencil(2 if gz > 1 else 1, gx, gy, gz, 1, seed=1)
    rng = np.random.default_rng(seed)
    return csr([[i] + [int(c) for c in ci[rp[i]:rp[i + 1]] if c != i and rng.random() < 0.7]
                for i in range(len(rp) - 1)])


def scattered(n, m, seed):
    rng = np.random.default_rng(seed)
    return csr([[i] + [int(c) for c in rng.integers(0, n, m)] for i in range(n)])


def batch(rp, ci, nsys, seed):
    rng = np.random.default_rng(seed)
    row = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    v = -rng.random((nsys, len(ci)))
    v[:, ci == row] += 1.1 * np.diff(rp).max()
    return v, rng.uniform(-1.0, 1.0, (nsys, len(rp) - 1))


SMALL = {
    "triangular_16x16": grid2d(16, 16, TRIANGULAR), "triangular_9x13": grid2d(9, 13, TRIANGULAR),
    "penta_300": band(300, (-2, -1, 1, 2)), "penta_1000": band(1000, (-2, -1, 1, 2)),
    "tri_513": band(513, (-1, 1)), "one_sided_17x15": one_sided(17, 15, 1, 1),
    "one_sided_7x6x5": one_sided(7, 6, 5, 2), "scattered_200": scattered(200, 1, 3),
    "scattered_700": scattered(700, 2, 4), "nine_20x20": grid2d(20, 20, NINE),
}


@pytest.mark.parametrize("name", list(SMALL))
@pytest.mark.parametrize("approach", [1, 2, 3, 4])
@pytest.mark.parametrize("nsys", [3, 2500])
def test_ilu0(cuda, name, approach, nsys):
    import torch
    rp, ci = SMALL[name]
    v, _ = batch(rp, ci, 3, 7)
    with bilu.Plan(rp, ci) as plan:
        V = torch.from_numpy(v).to(cuda).repeat(-(-nsys // 3), 1)[:nsys].contiguous()
        LU = torch.full_like(V, float("nan"))
        plan.ilu0(V, LU, approach)
        torch.cuda.synchronize()
    got = LU.cpu().numpy()
    want = O.ilu0(rp, ci, v, approach)
    H.assert_bitwise(got[:3], want, name)
    H.assert_bitwise(got[-1], want[(nsys - 1) % 3], name)


@pytest.mark.parametrize("name", list(SMALL))
@pytest.mark.parametrize("approach", [1, 2, 3])
@pytest.mark.parametrize("precond,fp32", [(bilu.PRECOND_ILU0, False), (bilu.PRECOND_ILU0, True),
                                          (bilu.PRECOND_PARILU0, False)])
def test_solves(cuda, name, approach, precond, fp32):
    rp, ci = SMALL[name]
    v, b = batch(rp, ci, 3, 8)
    kw = dict(precond=precond, ilu_approach=approach, factor_precision=bilu.FP32 if fp32 else bilu.FP64, **TOL)
    g = H.gpu_solve(cuda, rp, ci, v, b, **kw)
    o = H.oracle_pipeline(rp, ci, v, b, precond, approach=approach, fp32=fp32, **TOL)
    for f in FIELDS:
        H.assert_bitwise(g[f], o[f], f"{name}, reference order: {f}")
    g = H.gpu_solve(cuda, rp, ci, v, b, reduction=bilu.REDUCE_FAST, **kw)
    assert g["info"]["solver_kernel"] == 1
    o = H.oracle_fast(rp, ci, v, b, precond, g["info"]["threads"], fp32, approach=approach, **TOL)
    for f in FIELDS:
        H.assert_bitwise(g[f], o[f], f"{name}, FAST order: {f}")


LARGE = {
    "nine_33x33": grid2d(33, 33, NINE), "nine_40x32": grid2d(40, 32, NINE), "penta_1200": band(1200, (-2, -1, 1, 2)),
    "triangular_36x36": grid2d(36, 36, TRIANGULAR), "scattered_1100": scattered(1100, 8, 5),
    "scattered_1500": scattered(1500, 1, 6), "scattered_2048": scattered(2048, 3, 7),
}


@pytest.mark.parametrize("name", list(LARGE))
@pytest.mark.parametrize("precond,fp32", [(bilu.PRECOND_ILU0, False), (bilu.PRECOND_ILU0_SPLIT, True),
                                          (bilu.PRECOND_PARILU0, False), (bilu.PRECOND_PARILU0, True),
                                          (bilu.PRECOND_NONE, False)])
@pytest.mark.parametrize("nsys", [2, 400])
def test_large_systems(cuda, name, precond, fp32, nsys):
    """1025 to 2048 rows: rows of up to 16 entries, rows without upper entries, levels of one row and levels wider
    than a CTA; few systems and more than the GPU has SMs."""
    rp, ci = LARGE[name]
    v, b = batch(rp, ci, 2, 9)
    r = nsys // 2
    vs, bs = np.tile(v, (r, 1)), np.tile(b, (r, 1))
    kw = dict(precond=precond, factor_precision=bilu.FP32 if fp32 else bilu.FP64, **TOL)
    g = H.gpu_solve(cuda, rp, ci, vs, bs, **kw)
    o = H.oracle_pipeline(rp, ci, v, b, precond, fp32=fp32, **TOL)
    fast = dict(kw, reduction=bilu.REDUCE_FAST)
    q = H.gpu_solve(cuda, rp, ci, vs, bs, **fast)
    s = H.gpu_solve(cuda, rp, ci, v, b, threads_per_system=1024, **fast)
    assert g["info"]["solver_kernel"] == q["info"]["solver_kernel"] == 1 and s["info"]["solver_kernel"] == 0
    for f in FIELDS:
        H.assert_bitwise(g[f][:2], o[f], f"{name}, reference order: {f}")
        H.assert_bitwise(g[f][-2:], o[f], f"{name}, reference order: {f}, last systems")
        H.assert_bitwise(q[f][:2], s[f], f"{name}, FAST order: {f}")
        H.assert_bitwise(q[f][-2:], s[f], f"{name}, FAST order: {f}, last systems")
