"""The persistent launch's grid follows the graph's size: graphs on both sides
of its limits (1,572,864 and 5,242,880 vertices + edges), and one whose search
moves to the resume launch, one after the other on one context, so that every
change of grid between calls is met; ids against the oracle's Tarjan."""
import numpy as np
import pytest

import kaspan_b200 as K
import kaspan_b200.graphs as KG
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graphs(ctx):
    import torch

    rng = np.random.default_rng(11)
    out = []
    for n, m in ((30000, 30000), (24000, 1548863), (24000, 1548865), (200000, 5042879), (200000, 5042881)):
        if m == n:
            s, d = np.arange(n), np.roll(np.arange(n), -1)
        else:  # m distinct pairs without loops
            key = rng.choice(n * (n - 1), size=m, replace=False) if n < 30000 else np.unique(rng.integers(0, n * (n - 1), m + 10000))
            key = rng.permutation(key)[:m]
            s, d = key // (n - 1), key % (n - 1)
            d = d + (d >= s)
        G = KG.from_edges(ctx, n, *(torch.from_numpy(x.astype(np.int32)).cuda() for x in (s, d)))
        assert G.m == m
        fwh, fwc, bwh, bwc = G.to_host()
        out.append((G, O.tarjan(O.Graph(n, fwh, fwc, bwh, bwc))))
    return out


@pytest.mark.parametrize("order", [(0, 1, 2, 3, 4, 0), (4, 0, 3, 1, 4, 2), (1, 3, 0, 2, 0, 4)])
def test_grid_changes_between_calls(ctx, graphs, order):
    import torch

    for i in order:
        G, want = graphs[i]
        out = torch.empty(G.n, dtype=torch.int32, device="cuda")
        ctx.scc_device(G.n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options())
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
