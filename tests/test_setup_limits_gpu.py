"""ParILU(0) and ISAI in the reference order at the shared-memory limit, where
the diagonal's reciprocals no longer fit beside the iterates (ParILU) or the
ISAI values and the kernels divide instead: bit for bit against the oracle, on
both sides of the limit."""
import numpy as np
import pytest

import bilu
import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu


def _band(n, below, above, nsys, seed):
    rows = [list(range(max(0, i - below), min(n, i + above + 1))) for i in range(n)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    ci = np.concatenate(rows).astype(np.int32)
    rng = np.random.default_rng(seed)
    isd = ci == np.repeat(np.arange(n), np.diff(rp))
    v = np.where(isd[None, :], 2.0 + below + above + rng.random((nsys, len(ci))), -rng.random((nsys, len(ci))))
    return rp, ci, np.ascontiguousarray(v)


@pytest.mark.parametrize("n", [900, 990, 1010, 1035])
def test_parilu0_reference_order_near_the_limit(cuda, n):
    """Two iterates of 14 entries per row take 202 KB at n = 900 (reciprocals fit) and 231 KB at n = 1035 (they do
    not); sweeps with many pairs per entry."""
    import torch
    rp, ci, v = _band(n, 8, 5, 2, n)
    with bilu.Plan(rp, ci, precond=bilu.PRECOND_PARILU0) as plan:
        V = torch.from_numpy(v).to(cuda)
        LU = torch.empty_like(V)
        plan.parilu0(V, LU, 3)
        torch.cuda.synchronize()
    H.assert_bitwise(LU.cpu().numpy(), O.parilu0(rp, ci, v, 3), f"bilu_parilu0 n={n}")


@pytest.mark.parametrize("n", [900, 1030])
def test_isai_reference_order_near_the_limit(cuda, n):
    """aiU of 28 entries per row takes 202 KB at n = 900 (reciprocals fit) and 228 KB at n = 1030 (they do not)."""
    import torch
    rp, ci, lu = _band(n, 2, 27, 2, n)
    with bilu.Plan(rp, ci, precond=bilu.PRECOND_ILU0_ISAI, isai_power=1) as plan:
        i = plan.info()
        LU = torch.from_numpy(lu).to(cuda)
        AIL = torch.empty((2, i["nnz_isai_L"]), dtype=torch.float64, device=cuda)
        AIU = torch.empty((2, i["nnz_isai_U"]), dtype=torch.float64, device=cuda)
        plan.isai(LU, AIL, AIU)
        torch.cuda.synchronize()
    lrp, lci, urp, uci = O.split_pattern(rp, ci)
    L, U = O.split_values(rp, ci, lu)
    arp, aci = O.isai_pattern(lrp, lci, 1)
    brp, bci = O.isai_pattern(urp, uci, 1)
    H.assert_bitwise(AIL.cpu().numpy(), O.isai_values(lrp, lci, L, 0, arp, aci), f"aiL n={n}")
    H.assert_bitwise(AIU.cpu().numpy(), O.isai_values(urp, uci, U, 1, brp, bci), f"aiU n={n}")
