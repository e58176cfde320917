"""The training kernel's gradient and loss: the same bits on every run, for
batches of one block, of a part of a block, of one part of the blocks' rows and
of several, and the parts' sums against one another."""
import numpy as np
import pytest

import bilu
import helpers as H

pytestmark = pytest.mark.gpu


def _targets(cuda, nsys):
    import torch
    rp, ci, v, _ = bilu.gen_stencil(5, 7, 7, 7, nsys, seed=5)
    plan = bilu.Plan(rp, ci, precond=bilu.PRECOND_PARILU0)
    V = torch.from_numpy(v).to(cuda)
    LU = torch.empty_like(V)
    plan.parilu0(V, LU, 40)
    torch.cuda.synchronize()
    return plan, V, LU


@pytest.mark.parametrize("batch", [1, 127, 129, 20000, 65536, 200000])
def test_training_repeats_bit_for_bit(cuda, batch):
    plan, V, LU = _targets(cuda, 64)
    runs = []
    for _ in range(3):
        with bilu.Mlp(seed=1) as m:
            losses = m.train(plan, V, LU, 12, batch, 2e-3, seed=3)
            runs.append((losses, m.params()))
    assert np.all(np.isfinite(runs[0][0]))
    for losses, params in runs[1:]:
        H.assert_bitwise(losses, runs[0][0], f"losses, batch {batch}")
        H.assert_bitwise(params, runs[0][1], f"parameters, batch {batch}")
    plan.close()


def test_gradient_of_parts(cuda):
    """2^18 samples are more blocks than there are rows.  Scaled by powers of two, the blocks' shares are the same
    numbers in the whole batch and in its 16 parts, so the whole gradient is the parts' mean up to one rounding of
    each: half an ulp of the whole and of every part."""
    plan, V, LU = _targets(cuda, 64)
    idx = np.random.default_rng(2).integers(0, V.numel(), 1 << 18).astype(np.int32)
    with bilu.Mlp(seed=1) as m:
        m.train(plan, V, LU, 10, 4096, 2e-3, seed=1)
        loss, grad = m.loss_grad(plan, V, LU, idx)
        again = m.loss_grad(plan, V, LU, idx)
        parts = [m.loss_grad(plan, V, LU, p) for p in idx.reshape(16, -1)]
    H.assert_bitwise(again[1], grad, "gradient, second run")
    assert again[0] == loss
    g = np.array([np.append(p[1], np.float32(p[0])) for p in parts], np.float64)
    whole = np.append(grad, np.float32(loss)).astype(np.float64)
    bound = 2.0 ** -24 * 1.001 * (np.abs(whole) + np.abs(g).mean(0)) + 2.0 ** -140
    assert np.all(np.abs(whole - g.mean(0)) <= bound)
    plan.close()
