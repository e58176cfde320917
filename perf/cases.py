"""Performance cases of the batched solver library: what its users have it do.

A case goes through the public Python binding (merging-ilu0_gb300/bilu.py), as
a program does that keeps a plan for its sparsity pattern and calls the
library once per time step or Newton step with new values:

  solve    Plan.solve on a batch that shares one stencil pattern
  factor   the stand-alone factorisation and ISAI entry points
  uneven   UnevenPlan.solve: every system its own size and pattern
  learned  Mlp.warm_start, then Plan.solve from the predicted factors
  train    Mlp training from scratch: create, train, read the weights

Grids, value distributions, stopping rules and options are those of the
repository's benchmark and tests (families 1, 2, 4, 5 of bilu_gen_stencil, the
uneven generator's 5..12 off-diagonals per row); the values themselves are
drawn here with torch, on the GPU.

REF is the reference's operation order (the default options, what a program
re-linked from the reference's solvers gets: absolute tolerance 1e-11), FAST
the throughput order with a relative tolerance of 1e-10.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "merging-ilu0_gb300"))

import bilu  # noqa: E402

DEV = "cuda"
SOLVE_DEFAULTS = dict(kind="solve", order="fast", fp32=0, approach=1, sweeps=5, threads=0, staging=-1)


def listed():
    return [
        # The smallest call: a handful of cells of a 2D multiphysics code, default options (merged ILU(0),
        # reference order).  Launch and per-iteration latency are all there is.
        solve("ref_merged_2d8_few", 1, (8, 8, 1), 8, bilu.PRECOND_ILU0, order="ref"),
        # A few larger systems per step, fewer than the GPU has SMs: ParILU(5) + FP32 ISAI, default configuration.
        solve("isai32_3d10_few", 2, (10, 10, 10), 16, bilu.PRECOND_PARILU0_ISAI, fp32=1),
        # The reference's namesake solver on its benchmark pattern, bit for bit the reference's results.
        solve("ref_merged_2d16", 1, (16, 16, 1), 4096, bilu.PRECOND_ILU0, order="ref"),
        # The reference's ILU(0)-ISAI solver (serial inner products) as a re-linked program calls it.
        solve("ref_isai_2d16", 1, (16, 16, 1), 2048, bilu.PRECOND_ILU0_ISAI, order="ref", approach=3),
        # Systems past the 1024 rows of the register-resident kernels: ParILU(5) with triangular solves.
        solve("ref_parilu_2d36", 1, (36, 36, 1), 512, bilu.PRECOND_PARILU0, order="ref"),
        # The plain form at full size: merged FP64 ILU(0) of the benchmark's 3D systems.
        solve("ilu64_3d10", 2, (10, 10, 10), 4096, bilu.PRECOND_ILU0),
        # The benchmark's headline batch, in the configuration its autotuner keeps (256 threads, occupancy
        # variant), pinned because the FAST order depends on the threads per system.
        solve("isai32_3d10", 2, (10, 10, 10), 4096, bilu.PRECOND_PARILU0_ISAI, fp32=1, threads=256, staging=16),
        # The precision workload (convection-diffusion, ILU(0) + FP32 ISAI) on a ragged 23x25 grid; the largest.
        solve("isai32_cd23x25", 4, (23, 25, 1), 16384, bilu.PRECOND_ILU0_ISAI, fp32=1, approach=3),
        # Preconditioner generation on its own: ParILU(0) factors and their ISAI in the reference's arithmetic.
        dict(name="factor_isai_3d10", kind="factor", family=2, gx=10, gy=10, gz=10, nsys=1024, sweeps=5),
        # Uneven batch: n log-uniform in [64, 1024], random patterns, merged FP64 ILU(0), one graph launch.
        dict(name="uneven_64_1024", kind="uneven", nsys=2048, nmin=64, nmax=1024, fp32=0),
        # The learned warm start and adaptive ParILU on the 7x7x7 systems it is trained for, then the solve.
        dict(name="learned_3d7", kind="learned", family=5, gx=7, gy=7, gz=7, nsys=4096),
        # Training of the warm start's network: 40 steps of 65536 nonzeros from 2048 systems.
        dict(name="train_3d7", kind="train", family=5, gx=7, gy=7, gz=7, nsys=2048, steps=40, batch=65536),
    ]


def solve(name, family, grid, nsys, precond, **kw):
    return dict(SOLVE_DEFAULTS, name=name, family=family, gx=grid[0], gy=grid[1], gz=grid[2], nsys=nsys,
                precond=precond, **kw)


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(nmax):
        if rng.random() < 0.5:
            f = rng.choice([1, 4])
            m = int(math.isqrt(nmax))
            g = [rng.randint(6, m), rng.randint(6, m), 1]
        else:
            f = rng.choice([2, 5])
            m = int(round(nmax ** (1 / 3)))
            g = [rng.randint(4, m), rng.randint(4, m), rng.randint(4, m)]
        return f, g

    what = rng.choice(["fast", "fast", "fast", "ref", "ref", "refisai", "large", "factor", "uneven", "learned",
                       "train"])
    if what == "fast":  # throughput order: every preconditioner, both factor precisions, one system to a full batch
        f, g = grid(1000)
        n = g[0] * g[1] * g[2]
        p = rng.choice([bilu.PRECOND_ILU0, bilu.PRECOND_ILU0_SPLIT, bilu.PRECOND_PARILU0, bilu.PRECOND_ILU0_ISAI,
                        bilu.PRECOND_PARILU0_ISAI, bilu.PRECOND_PARILU0_ISAI])
        kw = dict(threads=-(-n // 128) * 32, staging=16) if rng.random() < 0.3 else {}
        c = solve("", f, g, logint(1, max(1, 4000000 // n)), p, fp32=rng.randint(0, 1), approach=rng.choice([1, 3]),
                  **kw)
    elif what == "ref":  # the reference's ILU solvers
        f, g = grid(1000)
        n = g[0] * g[1] * g[2]
        c = solve("", f, g, logint(1, max(1, 1000000 // n)),
                  rng.choice([bilu.PRECOND_ILU0, bilu.PRECOND_ILU0_SPLIT, bilu.PRECOND_PARILU0]), order="ref",
                  approach=rng.choice([1, 3]))
    elif what == "refisai":  # the reference's ISAI solvers
        f, g = grid(600)
        n = g[0] * g[1] * g[2]
        c = solve("", f, g, logint(1, max(1, 500000 // n)),
                  rng.choice([bilu.PRECOND_ILU0_ISAI, bilu.PRECOND_PARILU0_ISAI]), order="ref", approach=3)
    elif what == "large":  # past 1024 rows, up to what shared memory holds
        g = [rng.randint(33, 40), rng.randint(33, 40), 1]
        c = solve("", rng.choice([1, 4]), g, logint(1, 512),
                  rng.choice([bilu.PRECOND_ILU0_SPLIT, bilu.PRECOND_PARILU0]), order=rng.choice(["ref", "fast"]))
    elif what == "factor":
        f, g = grid(1000)
        c = dict(kind="factor", family=f, gx=g[0], gy=g[1], gz=g[2], nsys=logint(1, 1024), sweeps=rng.randint(2, 6))
    elif what == "uneven":
        lo = logint(32, 256)
        c = dict(kind="uneven", nsys=logint(4, 2048), nmin=lo, nmax=logint(2 * lo, 1024), fp32=rng.randint(0, 1))
    elif what == "learned":
        c = dict(kind="learned", family=5, gx=rng.randint(5, 8), gy=rng.randint(5, 8), gz=rng.randint(5, 8),
                 nsys=logint(1, 4096))
    else:
        c = dict(kind="train", family=5, gx=rng.randint(5, 8), gy=rng.randint(5, 8), gz=rng.randint(5, 8),
                 nsys=logint(16, 2048), steps=rng.randint(5, 40), batch=logint(1000, 65536))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- inputs (torch and numpy only)
class Pattern:
    """CSR pattern of a 2D 5-point / 3D 7-point stencil, columns ascending, with index arrays on the GPU."""

    def __init__(self, grid):
        gx, gy, gz = grid
        n = gx * gy * gz
        i = np.arange(n)
        x, y, z = i % gx, i // gx % gy, i // (gx * gy)
        cand = [(z > 0, -gx * gy), (y > 0, -gx), (x > 0, -1), (i >= 0, 0), (x < gx - 1, 1), (y < gy - 1, gx),
                (z < gz - 1, gx * gy)]
        ok = np.stack([c[0] for c in cand], 1)
        cols = np.stack([i + c[1] for c in cand], 1)
        self.n = n
        self.rp = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int32)
        self.ci = cols[ok].astype(np.int32)
        self.nnz = len(self.ci)
        self.row = np.repeat(i, np.diff(self.rp))
        self.pos = {(int(a), int(b)): k for k, (a, b) in enumerate(zip(self.row, self.ci))}
        self.diag = np.array([self.pos[(a, a)] for a in range(n)])

    def pairs(self):
        """(entry, l_ik, u_kj) of every product of (L U) on the pattern, k < min(i, j), k ascending."""
        e, l, u = [], [], []
        for k in range(self.nnz):
            i, j = int(self.row[k]), int(self.ci[k])
            for q in range(self.rp[i], self.rp[i + 1]):
                m = int(self.ci[q])
                if m >= min(i, j):
                    break
                p = self.pos.get((m, j))
                if p is not None:
                    e.append(k)
                    l.append(q)
                    u.append(p)
        return [torch.tensor(a, dtype=torch.int64, device=DEV) for a in (e, l, u)]


def gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def stencil_inputs(family, grid, nsys, seed):
    P = Pattern(grid)
    g = gen(seed)

    def u01(*shape):
        return torch.rand(*shape, generator=g, dtype=torch.float64, device=DEV)

    d = torch.tensor(P.ci.astype(np.int64) - P.row, device=DEV)
    pe = u01(nsys, 1)
    if family == 4:
        v = torch.where(d == 0, 4.0 + 2.0 * pe, torch.where(d == -1, -1.0 - 2.0 * pe, torch.full_like(pe, -1.0)))
    else:
        spread = {1: 0.2, 2: 0.25, 5: 0.3}[family]
        u = u01(nsys, P.nnz)
        v = torch.where(d == 0, (4.0 if family == 1 else 6.0) + u, -(1.0 + spread * (2.0 * u - 1.0)))
        if family == 1:
            skew = 0.3 * u01(nsys, P.n)[:, torch.tensor(P.row, device=DEV)]
        else:
            skew = 0.25 * pe if family == 2 else torch.zeros_like(pe)
        v = v + torch.where(d == 1, skew, torch.zeros_like(skew)) - torch.where(d == -1, skew, torch.zeros_like(skew))
    b = 2.0 * u01(nsys, P.n) - 1.0
    return P, v.contiguous(), b


def uneven_inputs(c, seed):
    """Systems back to back: sizes, local row pointers and columns (numpy), values and right-hand sides (GPU)."""
    rng = np.random.default_rng(seed)
    nsys = c["nsys"]
    u = np.random.default_rng(nsys).random(nsys)  # the sizes belong to the program, patterns and values to the seed
    sn = np.exp(math.log(c["nmin"]) + u * math.log((c["nmax"] + 1) / c["nmin"])).astype(np.int64)
    sn = np.clip(sn, c["nmin"], c["nmax"])
    n_row = np.repeat(sn, sn)
    off = np.concatenate([[0], np.cumsum(sn)])
    i_row = np.arange(off[-1]) - np.repeat(off[:-1], sn)
    k = rng.integers(5, 13, off[-1])
    cols = (rng.random((off[-1], 13)) * n_row[:, None]).astype(np.int64)
    cols[np.arange(13)[None, :] >= k[:, None]] = 1 << 40
    cols[:, 12] = i_row
    cols.sort(1)
    keep = cols < (1 << 40)
    keep[:, 1:] &= cols[:, 1:] != cols[:, :-1]
    ci = cols[keep]
    rlen = keep.sum(1)
    ends = np.cumsum(rlen)
    sz = ends[off[1:] - 1] - np.concatenate([[0], ends[off[1:-1] - 1]])
    rp = np.insert(ends - np.repeat(np.concatenate([[0], np.cumsum(sz)[:-1]]), sn), off[:-1], 0)
    row = np.repeat(np.arange(off[-1]), rlen)
    v = rng.standard_normal(len(ci))
    isd = ci == i_row[row]
    v[isd] = 0.0
    rsum = np.bincount(row, np.abs(v), minlength=off[-1])
    v[isd] = (1.2 * rsum * rng.choice([-1.0, 1.0], off[-1]))
    v[isd & (v == 0.0)] = 1.0
    b = rng.uniform(-1.0, 1.0, off[-1])
    i32 = np.int32
    return (sn.astype(i32), sz.astype(i32), rp.astype(i32), ci.astype(i32), torch.from_numpy(v).to(DEV),
            torch.from_numpy(b).to(DEV))


# ---------------------------------------------------------------- the learned part in 64 bits
def bf16(w):
    return w.to(torch.bfloat16).to(torch.float64)


def features(P, v):
    """Entry features (nsys, nnz, 9) and first-order factor estimates of the warm start, in 64 bits."""
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.int64, device=DEV)  # noqa: E731
    row, col, diag = t(P.row), t(P.ci), t(P.diag)
    tp = t([P.pos[(int(j), int(i))] for i, j in zip(P.row, P.ci)])
    lev = np.zeros(P.n)
    for i in range(P.n):
        lo = P.ci[P.rp[i]:P.diag[i]]
        lev[i] = lev[lo].max() + 1 if len(lo) else 0
    z = torch.zeros(v.shape[0], P.n, dtype=torch.float64, device=DEV)
    rn = z.index_add(1, row, v * v).sqrt()
    cn = z.index_add(1, row, v[:, tp] ** 2).sqrt()
    low = (col < row).to(torch.float64)
    cr = z.index_add(1, row, low * v * v[:, tp] / v[:, diag[col]])
    inv = 1.0 / v[:, diag[row]].abs()
    ii, jj, ci, cj = v[:, diag[row]], v[:, diag[col]], cr[:, row], cr[:, col]
    lv = torch.as_tensor(lev / max(lev.max(), 1), device=DEV)[row].expand_as(v)
    sg = torch.sign(col - row).to(torch.float64).expand_as(v)
    f = torch.stack([v * inv, ii * inv, jj * inv, rn[:, row] * inv, cn[:, col] * inv, lv, sg, ci * inv, cj * inv], 2)
    base = torch.where(col < row, 1.0 / (jj - cj), torch.where(col == row, (ii - ci) / ii, torch.ones_like(v)))
    return f, base


def gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def hidden(params, f):
    w1, b1, w2, b2 = (bf16(params[a:b]) for a, b in ((0, 576), (576, 640), (640, 4736), (4736, 4800)))
    h = gelu(f @ w1.view(64, 9).T + b1)
    return gelu(h @ w2.view(64, 64).T + b2)


_net = {}


def network():
    """Weights of the warm start's network, the same in every program: random hidden layers and an output layer
    fitted by least squares to the converged ParILU(0) factors of 48 7x7x7 systems."""
    if "p" not in _net:
        P, v, _ = stencil_inputs(5, (7, 7, 7), 48, 76)
        lu = parilu_exact(P, v, 40)
        f, base = features(P, v)
        low = torch.tensor(P.ci <= P.row, device=DEV)
        f = f[:, low].reshape(-1, 9)
        p = torch.randn(4865, generator=torch.Generator().manual_seed(78), dtype=torch.float64).to(DEV)
        w1 = 0.25 * p[:576].view(64, 9) / f.std(0).clamp_min(1e-2)
        p[576:640] = 0.5 * p[576:640] - w1 @ f.mean(0)
        p[:576] = w1.flatten()
        p[640:4736] *= 0.25
        h = hidden(p, f)
        h = torch.cat([h, torch.ones_like(h[:, :1])], 1)
        y = (lu / (v * base) - 1.0)[:, low].flatten()
        g = h.T @ h
        g += 1e-7 * g.diagonal().mean() * torch.eye(65, dtype=torch.float64, device=DEV)
        p[4800:] = torch.linalg.solve(g, h.T @ y)
        _net["p"] = p.float().cpu().numpy()
    return _net["p"]


# ---------------------------------------------------------------- prepare and run
def out_arrays(nsys, n_x):
    e = lambda dt, m: torch.empty(m, dtype=dt, device=DEV)  # noqa: E731
    return dict(x=e(torch.float64, n_x), iters=e(torch.float32, nsys), conv=e(torch.int32, nsys),
                res=e(torch.float64, nsys), true_res=e(torch.float64, nsys), status=e(torch.int32, nsys))


def grid_of(case):
    return case["gx"], case["gy"], case["gz"]


def prepare(case, seed):
    k = case["kind"]
    s = dict(kind=k, case=case)
    nsys = case["nsys"]
    if k == "uneven":
        sn, sz, rp, ci, s["V"], s["B"] = uneven_inputs(case, seed)
        s["plan"] = bilu.UnevenPlan(sn, sz, rp, ci, precond=bilu.PRECOND_ILU0, reduction=bilu.REDUCE_FAST,
                                    tol_mode=bilu.TOL_REL, tol=1e-10, factor_precision=case["fp32"])
        s["out"] = out_arrays(nsys, int(sn.sum()))
        return s
    P, s["V"], s["B"] = stencil_inputs(case["family"], grid_of(case), nsys, seed)
    s["out"] = out_arrays(nsys, (nsys, P.n))
    fast = dict(reduction=bilu.REDUCE_FAST, tol_mode=bilu.TOL_REL, tol=1e-10)
    if k == "solve":
        s["plan"] = bilu.Plan(P.rp, P.ci, precond=case["precond"], ilu_approach=case["approach"],
                              parilu_sweeps=case["sweeps"], factor_precision=case["fp32"],
                              threads_per_system=case["threads"], smem_staging=case["staging"],
                              **(fast if case["order"] == "fast" else {}))
    elif k == "factor":
        s["plan"] = p = bilu.Plan(P.rp, P.ci, precond=bilu.PRECOND_PARILU0_ISAI)
        i = p.info()
        for name, m in (("lu", i["nnz"]), ("ail", i["nnz_isai_L"]), ("aiu", i["nnz_isai_U"])):
            s[name] = torch.empty(nsys, m, dtype=torch.float64, device=DEV)
    elif k == "learned":
        s["plan"] = bilu.Plan(P.rp, P.ci, precond=bilu.PRECOND_PARILU0_ISAI, parilu_sweeps=40, parilu_res_tol=1e-6,
                              factor_precision=bilu.FP32, **fast)
        s["mlp"] = bilu.Mlp(seed=1)
        s["mlp"].set_params(network())
        s["lu0"] = torch.empty_like(s["V"])
        s["sweeps"] = torch.empty(nsys, dtype=torch.int32, device=DEV)
        s["used"] = torch.empty(nsys, dtype=torch.int32, device=DEV)
    else:
        s["plan"] = bilu.Plan(P.rp, P.ci, precond=bilu.PRECOND_PARILU0)
        s["lu"] = torch.empty_like(s["V"])
        s["plan"].parilu0(s["V"], s["lu"], 40)
    return s


def run(s):
    k, c, plan = s["kind"], s["case"], s["plan"]
    o = s["out"]
    if k in ("solve", "uneven"):
        plan.solve(s["V"], s["B"], o["x"], o["iters"], o["conv"], o["res"], o["true_res"], o["status"])
        return o
    if k == "factor":
        plan.parilu0(s["V"], s["lu"], c["sweeps"])
        plan.isai(s["lu"], s["ail"], s["aiu"])
        return dict(lu=s["lu"], ail=s["ail"], aiu=s["aiu"])
    if k == "learned":
        s["mlp"].warm_start(plan, s["V"], s["lu0"], 1e-3, None, s["used"])
        plan.solve(s["V"], s["B"], o["x"], o["iters"], o["conv"], o["res"], o["true_res"], o["status"],
                   lu_init=s["lu0"], sweeps=s["sweeps"])
        return dict(o, lu0=s["lu0"], used=s["used"], sweeps=s["sweeps"])
    with bilu.Mlp(seed=1) as m:
        losses = m.train(plan, s["V"], s["lu"], c["steps"], c["batch"], 2e-3, seed=3)
        return dict(losses=losses, params=m.params())


# ---------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once; FP64 operations of the method at its usual iteration counts."""
    k, nsys = case["kind"], case["nsys"]
    if k == "uneven":
        n = (case["nmax"] - case["nmin"]) / max(math.log(case["nmax"] / case["nmin"]), 1e-9)
        nnz = 9.4 * n
        it, prec, setup = 5.0, nnz, 4.0 * nnz
    else:
        gx, gy, gz = grid_of(case)
        n = gx * gy * gz
        nnz = n + 2 * ((gx - 1) * gy * gz + gx * (gy - 1) * gz + gx * gy * (gz - 1))
        isai = 2.1 * nnz if gz > 1 else 1.7 * nnz  # entries of aiL and aiU
        if k == "factor":
            return dict(bytes=8.0 * nsys * (2 * nnz + isai), flops=nsys * (case["sweeps"] * 2.0 * nnz + 4.0 * isai))
        if k == "train":
            per = 2.0 * (9 * 64 + 64 * 64 + 64) * 3
            return dict(bytes=16.0 * nsys * nnz + 4865 * 4.0, flops=per * case["steps"] * case["batch"])
        p = case.get("precond", bilu.PRECOND_PARILU0_ISAI)
        with_isai = p in (bilu.PRECOND_ILU0_ISAI, bilu.PRECOND_PARILU0_ISAI)
        it = 12.0 if n > 1024 else (9.5 if gz > 1 or n <= 256 else 14.0)
        prec = (isai if with_isai else nnz) * (0.0 if case.get("fp32", 1) else 1.0)  # FP64 products of one apply
        setup = (2.0 * nnz * case.get("sweeps", 5)) + (4.0 * isai if with_isai else 0.0)
    fma = it * (2 * nnz + 2 * prec + 11 * n) + setup / 2 + nnz
    return dict(bytes=nsys * (8.0 * nnz + 16.0 * n + 28.0) + (8.0 * nsys * nnz if k == "learned" else 0.0),
                flops=2.0 * nsys * fma)


# ---------------------------------------------------------------- the same in 64 bits, without the library
def solve_exact(P, grid, v, b):
    """x of every system by block elimination over the grid's lines (2D) or planes (3D)."""
    m = grid[0] if grid[2] == 1 else grid[0] * grid[1]
    nb = P.n // m
    out = torch.empty_like(b)
    step = max(1, int(2e9 // (8 * (nb + 3) * m * m)))
    row, col = (torch.as_tensor(a.astype(np.int64), device=DEV) for a in (P.row, P.ci))
    for s in range(0, v.shape[0], step):
        vs, bs = v[s:s + step], b[s:s + step]
        C, y = [], []
        for k in range(nb):
            def block(kk):
                sel = ((row // m == k) & (col // m == kk)).nonzero().flatten()
                M = torch.zeros(vs.shape[0], m * m, dtype=torch.float64, device=DEV)
                M[:, row[sel] % m * m + col[sel] % m] = vs[:, sel]
                return M.view(-1, m, m)
            D, r = block(k), bs[:, k * m:(k + 1) * m, None]
            if k:
                L = block(k - 1)
                D, r = D - L @ C[-1], r - L @ y[-1]
            R = torch.linalg.solve(D, torch.cat([r, block(k + 1)], 2) if k + 1 < nb else r)
            y.append(R[:, :, :1])
            C.append(R[:, :, 1:])
        x = y[-1]
        out[s:s + step, (nb - 1) * m:] = x[:, :, 0]
        for k in range(nb - 2, -1, -1):
            x = y[k] - C[k] @ x
            out[s:s + step, k * m:(k + 1) * m] = x[:, :, 0]
    return out


def parilu_exact(P, v, sweeps, init=None):
    e, l, u = P.pairs()
    low = torch.tensor(P.ci < P.row, device=DEV)
    dj = torch.tensor(P.diag[P.ci].astype(np.int64), device=DEV)
    lu = v.clone() if init is None else init.clone()
    for _ in range(sweeps):
        a = (v - torch.zeros_like(v).index_add_(1, e, lu[:, l] * lu[:, u])) if len(e) else v
        lu = torch.where(low, a / lu[:, dj], a)
    return lu


def isai_exact(P, lu, upper):
    """Row i of the inverse of L (unit diagonal) or U on the pattern of its square: m T(J,J) = e_i."""
    tri = [[int(c) for c in P.ci[P.rp[i]:P.rp[i + 1]] if (c >= i if upper else c <= i)] for i in range(P.n)]
    J = [sorted({c for q in tri[i] for c in tri[q]}) for i in range(P.n)]
    if not upper:  # solve from the diagonal outwards: columns descending
        J = [j[::-1] for j in J]
    s = max(map(len, J))
    # position of T(J_c, J_t) in lu; nnz: an exact 0, nnz + 1: an exact 1
    pos = np.full((P.n, s, s), P.nnz, np.int64)
    for i, j in enumerate(J):
        for t in range(s):
            pos[i, t, t] = P.nnz + 1 if t >= len(j) or not upper else P.pos[(j[t], j[t])]
            for c in range(min(t, len(j))):
                if t < len(j):
                    pos[i, c, t] = P.pos.get((j[c], j[t]), P.nnz)
    pos = torch.as_tensor(pos, device=DEV)
    ext = torch.cat([lu, torch.zeros_like(lu[:, :1]), torch.ones_like(lu[:, :1])], 1)
    m = torch.zeros(lu.shape[0], P.n, s, dtype=torch.float64, device=DEV)
    m[:, :, 0] = 1.0 / ext[:, pos[:, 0, 0]]
    for t in range(1, s):
        acc = torch.zeros_like(m[:, :, 0])
        for c in range(t):
            acc -= m[:, :, c] * ext[:, pos[:, c, t]]
        m[:, :, t] = acc / ext[:, pos[:, t, t]]
    order = torch.as_tensor(np.concatenate([i * s + np.argsort(j) for i, j in enumerate(J)]), device=DEV)
    return m.view(lu.shape[0], -1)[:, order]


def uneven_exact(case, seed):
    sn, sz, rp, ci, v, b = uneven_inputs(case, seed)
    ro = np.concatenate([[0], np.cumsum(sn.astype(np.int64))])
    zo = np.concatenate([[0], np.cumsum(sz.astype(np.int64))])
    x = torch.empty_like(b)
    order = np.argsort(sn, kind="stable")
    for g in range(0, len(sn), 64):
        ids = order[g:g + 64]
        m = int(sn[ids].max())
        A = torch.zeros(len(ids), m, m, dtype=torch.float64, device=DEV)
        r = torch.zeros(len(ids), m, 1, dtype=torch.float64, device=DEV)
        for q, i in enumerate(ids):
            n = int(sn[i])
            row = np.repeat(np.arange(n), np.diff(rp[ro[i] + i:ro[i] + i + n + 1]))
            flat = torch.from_numpy(row * m + ci[zo[i]:zo[i + 1]]).to(DEV)
            A[q].view(-1)[flat] = v[zo[i]:zo[i + 1]]
            A[q].view(-1)[n * (m + 1)::m + 1] = 1.0
            r[q, :n, 0] = b[ro[i]:ro[i + 1]]
        sol = torch.linalg.solve(A, r)
        for q, i in enumerate(ids):
            x[ro[i]:ro[i + 1]] = sol[q, :int(sn[i]), 0]
    return x


def warm_exact(P, v):
    """The predicted factors, A's own values where their ILU residual is above 1e-3."""
    p = torch.as_tensor(network(), device=DEV)
    e, l, u = P.pairs()
    pred = torch.tensor(P.ci < P.row, device=DEV)
    pred[e] = True
    dj = torch.tensor(P.diag[P.ci].astype(np.int64), device=DEV)
    low = torch.tensor(P.ci < P.row, device=DEV)
    out = torch.empty_like(v)
    step = max(1, int(4e8 // (P.nnz * 64 * 8)))
    for s in range(0, v.shape[0], step):
        vs = v[s:s + step]
        f, base = features(P, vs)
        y = hidden(p, f) @ bf16(p[4800:4864]) + bf16(p[4864:])
        lu = torch.where(pred, vs * base * (1.0 + y), vs)
        a = vs - (torch.zeros_like(vs).index_add_(1, e, lu[:, l] * lu[:, u]) if len(e) else 0.0)
        r = torch.where(low, a - lu * lu[:, dj], a - lu)
        bad = r.norm(dim=1) > 1e-3 * vs.norm(dim=1)
        out[s:s + step] = torch.where(bad[:, None], vs, lu)
    return out


def exact(case, seed):
    k = case["kind"]
    none = dict(x=None, iters=None, conv=None, res=None, true_res=None, status=None)
    if k == "train":
        return None  # the minibatches are drawn inside the call
    if k == "uneven":
        return dict(none, x=uneven_exact(case, seed))
    P, v, b = stencil_inputs(case["family"], grid_of(case), case["nsys"], seed)
    if k == "factor":
        lu = parilu_exact(P, v, case["sweeps"])
        return dict(lu=lu, ail=isai_exact(P, lu, False), aiu=isai_exact(P, lu, True))
    x = solve_exact(P, grid_of(case), v, b)
    if k == "learned":
        return dict(none, x=x, lu0=warm_exact(P, v), used=None, sweeps=None)
    return dict(none, x=x)
