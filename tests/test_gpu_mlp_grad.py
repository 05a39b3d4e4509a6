"""The gradient kernel at the edges of its work split (12 samples per block
and step, 148 blocks, at least four per warp) against the numpy restatement."""
import numpy as np
import pytest

import kaspan_b200 as K
import mlp as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 11, 12, 13, 47, 48, 49, 95, 97, 7103, 7104, 7105, 20001])
def test_gradient_sizes(ctx, n):
    import torch

    rng = np.random.default_rng(n)
    params = (rng.standard_normal(K.MLP_PARAMS) * 0.3).astype(np.float32)
    x = rng.uniform(0, 1.2, (n, 8)).astype(np.float32)
    y = rng.random(n).astype(np.float32)
    dp, dx, dy = (torch.from_numpy(a).cuda() for a in (params, x, y))
    g = torch.full((K.MLP_PARAMS,), 7.0, dtype=torch.float32, device="cuda")
    loss = torch.full((1,), 7.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    ctx.mlp_gradient(dx, dy, dp, g, loss)
    want_loss, want = M.loss_and_grad(params, x.astype(np.float64), y.astype(np.float64))
    # FP32 with at most 20001 / 1776 + 12 + 148 adds in a chain and 72 terms per
    # sample, each to 2^-24: under 250 * 6e-8 = 1.5e-5 of the terms' sizes, which
    # are at most 1 (dz) x 1.2 (x) x the weights along a path (below 4 here)
    assert abs(loss.item() - want_loss) <= 1.5e-5 * max(1.0, abs(want_loss))
    np.testing.assert_allclose(g.cpu().numpy(), want, rtol=1e-4, atol=5e-5)
