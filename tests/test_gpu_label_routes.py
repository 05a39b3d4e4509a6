"""Label searches on either side of the one-block limits, shown by the number
of launches: a leftover ring of 600 vertices needs 600 levels, each at least
one launch on the general path and none of its own in one block.  Every case
holds that ring and one piece that meets a limit exactly or passes it by one;
ids against the oracle's Tarjan."""
import numpy as np
import pytest

import kaspan_b200 as K
import kaspan_b200.graphs as KG
import oracle as O

pytestmark = pytest.mark.gpu

VERTICES, ENTRIES, ROW, RING = 1 << 15, 1 << 20, 8192, 600
CORE = 5000


def piece(kind, over):
    """(vertices, sources, targets) of the piece, local ids."""
    if kind == "vertices":
        k = VERTICES - RING + over
        i = np.arange(k)
        c = np.arange(1, 10)  # nine chords each: few levels
        return k, np.repeat(i, 9), (i[:, None] + c * 3001 % k).ravel() % k
    if kind == "entries":  # out- and in-rows of 22 entries, the ring's 2 x 600
        k = (ENTRIES // 2 - RING) // 22
        assert 2 * (22 * k + RING) == ENTRIES
        i = np.arange(k)
        s, d = np.repeat(i, 22), (i[:, None] + np.arange(1, 23)).ravel() % k
        return k, np.concatenate([s, [0] * over]), np.concatenate([d, [k // 2] * over])
    k = ROW + 500  # a ring with one long row
    i = np.arange(k)
    return k, np.concatenate([i, np.zeros(ROW - 1 + over, int)]), np.concatenate([np.roll(i, -1), np.arange(2, ROW + 1 + over)])


@pytest.mark.parametrize("mirror", [False, True])
@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("kind", ["vertices", "entries", "row"])
def test_limits(ctx, kind, over, mirror):
    import torch

    rng = np.random.default_rng(3)
    core = np.arange(CORE)
    k, ps, pd = piece(kind, over)
    ring = CORE + k + np.arange(RING)
    # the pivot: 200 edges each way, more in * out than any row of the piece
    e = [(core, np.roll(core, -1)), (np.zeros(200, int), rng.choice(core[1:], 200, replace=False)), (rng.choice(core[1:], 200, replace=False), np.zeros(200, int)),
         (CORE + ps, CORE + pd), (ring, np.roll(ring, -1))]
    s, d = (np.concatenate([x[i] for x in e]) for i in (0, 1))
    if mirror:
        s, d = d, s
    n = CORE + k + RING
    G = KG.from_edges(ctx, n, *(torch.from_numpy(x.astype(np.int32)).cuda() for x in (s, d)))
    assert G.m == len(np.unique(s * n + d))
    fwh, fwc, bwh, bwc = G.to_host()
    want = O.tarjan(O.Graph(n, fwh, fwc, bwh, bwc))
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    for pipeline in (K.PIPELINE_FAST, K.PIPELINE_REFERENCE, K.PIPELINE_HPC_LIKE, K.PIPELINE_TRIM_EX):
        st = K.Stats()
        ctx.scc_device(n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options(pipeline=pipeline), st)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        got = st.as_dict()
        assert want[got["pivot"]] == want[0] and got["label_calls"] >= 1
        assert (got["kernel_launches"] >= RING) == bool(over)
