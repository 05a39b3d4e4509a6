"""The searches' first levels in one block (graphs above the one-block size
whose largest in * out vertex has few neighbours): every way such an opening
ends -- a level that widens by its vertices or by one long row, exactly at the
limit of 512 entries, a search that runs dry, the level cap, the level the
worklist may start at -- with ids against the oracle's Tarjan and counts against the path with the opening switched off (the barrier hook set past the
launch's last barrier)."""
import numpy as np
import pytest

import kaspan_b200 as K
import kaspan_b200.graphs as KG
import oracle as O

pytestmark = pytest.mark.gpu

N = 30000


def tree_core(width, depth, seed):
    """From a root: `depth` levels that grow by `width`, mirrored backwards to
    the root, then a ring of the rest so that the graph is not small."""
    rng = np.random.default_rng(seed)
    s, d, level, nxt = [], [], np.array([0]), 1
    for _ in range(depth):
        kids = np.arange(nxt, nxt + len(level) * width)
        nxt += len(kids)
        s += [np.repeat(level, width), kids]
        d += [kids, rng.choice(level, len(kids))]  # back edges: all one component
        level = kids
    rest = np.arange(nxt, N)
    s, d = np.concatenate(s + [rest]), np.concatenate(d + [np.roll(rest, -1)])
    return s, d


def edges(kind):
    rng = np.random.default_rng(7)
    if kind == "random 2":
        return rng.integers(0, N, 2 * N), rng.integers(0, N, 2 * N)
    if kind == "random 8":
        return rng.integers(0, N, 8 * N), rng.integers(0, N, 8 * N)
    if kind == "near threshold":
        return rng.integers(0, N, int(1.1 * N)), rng.integers(0, N, int(1.1 * N))
    if kind == "ring":
        return np.arange(N), np.roll(np.arange(N), -1)
    if kind == "long row next":  # the pivot (20 x 20) leads to one row of 9,000
        a = np.arange(100, 120)
        out = np.arange(1000, 10000)
        return (np.concatenate([np.zeros(20, int), a, a, np.full(9000, 50), [out[0]], np.arange(20000, N)]),
                np.concatenate([a, np.zeros(20, int), np.full(20, 50), out, [0], np.roll(np.arange(20000, N), -1)]))
    if kind == "512":  # two levels of 2 x 256 entries each way, then wider
        return tree_core(8, 4, 1)
    if kind == "dry":  # the pivot's component is 41 vertices
        a = np.arange(1, 41)
        return np.concatenate([np.zeros(40, int), a, np.arange(100, N)]), np.concatenate([a, np.zeros(40, int), np.roll(np.arange(100, N), -1)])
    return tree_core(2, 11, 2)


@pytest.mark.parametrize("kind", ["random 2", "random 8", "near threshold", "ring", "long row next", "512", "dry", "binary"])
def test_opening_matches(ctx, kind):
    import torch

    s, d = edges(kind)
    G = KG.from_edges(ctx, N, *(torch.from_numpy(x.astype(np.int32)).cuda() for x in (s, d)))
    fwh, fwc, bwh, bwc = G.to_host()
    want = O.tarjan(O.Graph(N, fwh, fwc, bwh, bwc))
    out = torch.empty(N, dtype=torch.int32, device="cuda")
    res = []
    for drop in (0, 1 << 20):
        st = K.Stats()
        ctx.scc_device(G.n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options(drop_barrier=drop), st)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        res.append(st.as_dict())
    assert res[0]["kernel_launches"] == res[1]["kernel_launches"]
    assert res[0]["pivot"] == res[1]["pivot"] and res[0]["decided"] == res[1]["decided"]


def test_level_cap(ctx):
    """max_levels below, at and above the opening's length is met as before."""
    import torch

    s, d = edges("ring")
    G = KG.from_edges(ctx, N, *(torch.from_numpy(x.astype(np.int32)).cuda() for x in (s, d)))
    out = torch.empty(N, dtype=torch.int32, device="cuda")
    for cap in (1, 2, 7, 8, 9, 12):
        with pytest.raises(K.KspnError) as e:
            ctx.scc_device(G.n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options(max_levels=cap))
        assert e.value.status == 4
    ctx.scc_device(G.n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options())
    assert (out.cpu().numpy() == 0).all()
