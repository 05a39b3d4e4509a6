"""The searches' first levels in one block: the trace shows whether they ran
(phase 18, their end), so that a dispatch that never takes them fails."""
import numpy as np
import pytest

import kaspan_b200 as K
import kaspan_b200.graphs as KG

pytestmark = pytest.mark.gpu

HANDED_OVER = 18


def phases(ctx, G, **kw):
    import torch

    st = K.Stats()
    out = torch.empty(G.n, dtype=torch.int32, device="cuda")
    ctx.scc_device(G.n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options(trace=1, **kw), st)
    return [p for p, _ in st.as_dict()["search_marks"]]


@pytest.mark.parametrize("n,degree", [(30000, 2), (30000, 8), (300001, 1.1), (1 << 20, 3)])
def test_opening_runs(ctx, n, degree):
    G = KG.gnm(ctx, n, int(n * degree), 5)
    got = phases(ctx, G)
    assert got.count(HANDED_OVER) == 1 and got.index(HANDED_OVER) >= 3  # launch start, init, at least one level
    assert HANDED_OVER not in phases(ctx, G, drop_barrier=1 << 20)  # the hook keeps it off


def test_wide_first_level_takes_the_grid(ctx):
    """A pivot with more entries than the opening's 512 starts grid-wide."""
    import torch

    n = 30000
    rng = np.random.default_rng(1)
    hub = np.zeros(600, int)
    a, b = (rng.choice(np.arange(1, n), 600, replace=False) for _ in range(2))
    s, d = np.concatenate([np.arange(n), hub, a]), np.concatenate([np.roll(np.arange(n), -1), b, hub])
    G = KG.from_edges(ctx, n, *(torch.from_numpy(x.astype(np.int32)).cuda() for x in (s, d)))
    assert HANDED_OVER not in phases(ctx, G)
