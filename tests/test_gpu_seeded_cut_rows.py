"""Bottom-up sweeps that leave a heavy row open before the worklist phase: a
hub of the pivot's component whose row starts with 3000 vertices the search
never reaches is on the cut list, reached by neither or only one search, when
a long thin tail moves both to the worklist -- on a graph of enough vertices
for several start vertices, some of them outside the component.  The hub, and
what only it leads to, belong to the component all the same.  Output
bit-identical to the oracle's Tarjan."""
from __future__ import annotations

import numpy as np
import pytest

import kaspan_b200 as K
import kaspan_b200.graphs as KG
import oracle as O
from test_gpu_seeded_search import build

pytestmark = pytest.mark.gpu

HUB, CORE, CHAIN, APART, N = 3000, 3001, 23001, 26001, 40001


def edges(beyond):
    """Sources 0 .. HUB - 1 -> the hub; a dense core with the pivot; the core's
    last vertex -> the hub -> the core, with `beyond` by way of that many
    further vertices; a chain out of the core and back; cycles of 1000 apart."""
    rng = np.random.default_rng(1)
    core, chain = np.arange(CORE, CHAIN), np.arange(CHAIN, APART)
    if beyond:
        chain, more = chain[:-beyond], chain[-beyond:]
    e = [(np.arange(HUB), np.full(HUB, HUB)), (core, np.roll(core, -1))]
    e.append((rng.choice(core, 20 * len(core)), rng.choice(core, 20 * len(core))))
    pivot = core[500]
    e += [(np.full(100, pivot), rng.choice(core, 100)), (rng.choice(core, 100), np.full(100, pivot))]
    e.append((core[-1:], [HUB]))
    path = np.concatenate([[HUB], more, core[:1]]) if beyond else np.array([HUB, core[0]])
    e.append((path[:-1], path[1:]))
    loop = np.concatenate([core[700:701], chain, core[9000:9001]])
    e.append((loop[:-1], loop[1:]))
    for first in range(APART, N, 1000):
        ring = np.arange(first, min(first + 1000, N))
        e.append((ring, np.roll(ring, -1)))
    s, d = (np.concatenate([np.asarray(x[i]) for x in e]) for i in (0, 1))
    return s.astype(np.uint32), d.astype(np.uint32), pivot


@pytest.mark.parametrize("validate", [0, 1])
@pytest.mark.parametrize("mirror", [False, True])
@pytest.mark.parametrize("beyond", [0, 1, 100])
def test_hub_on_the_cut_list(ctx, beyond, mirror, validate):
    import torch

    s, d, pivot = edges(beyond)
    if mirror:
        s, d = d, s
    G = KG.from_edges(ctx, N, *(torch.from_numpy(x.view(np.int32)).cuda() for x in (s, d)))
    fwh, fwc, bwh, bwc = G.to_host()
    want = O.tarjan(O.Graph(N, fwh, fwc, bwh, bwc))
    assert want[HUB] == want[pivot] and want[APART] != want[pivot]
    out = torch.empty(N, dtype=torch.int32, device="cuda")
    for after in (0, 1):  # the worklist's two take policies, and its state after a call
        st = K.Stats()
        ctx.scc_device(N, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options(validate=validate, aw_exact_after=after), st)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        got = st.as_dict()
        assert got["pivot"] == pivot
        assert got["heavy"]["cut_rows"] > 0 and got["search_worklist"] == 1


@pytest.mark.parametrize("mirror", [False, True])
@pytest.mark.parametrize("kind", ["upstream", "both", "through"])
def test_rows_cut_after_the_restart(ctx, kind, mirror):
    """Thin from the first level on, so no sweep comes before the start
    vertices; some of them outside the component, so that both sets restart
    and sweep; hubs on the component's cycle behind 3000 sources each, whose
    rows those sweeps cut."""
    import torch

    n0, s, d = build(kind)
    first, hubs = 3 * HUB, (23000, 61000, 90500)  # the sources' ids come first in the hubs' rows
    pivot = first + np.bincount(s, minlength=n0).argmax()
    rng = np.random.default_rng(5)
    main = np.flatnonzero(np.bincount(s, minlength=n0) == 1) + first
    e = [(s.astype(np.int64) + first, d.astype(np.int64) + first)]
    for i, h in enumerate(hubs):
        e.append((np.arange(i * HUB, (i + 1) * HUB), np.full(HUB, main[np.searchsorted(main, h)])))
    fan = rng.choice(main[1000:2000], 100, replace=False)  # more in * out than a hub's 3001 x 1
    e += [(np.full(100, pivot), fan), (fan, np.full(100, pivot))]
    s, d = (np.concatenate([x[i] for x in e]).astype(np.uint32) for i in (0, 1))
    if mirror:
        s, d = d, s
    n = n0 + first
    G = KG.from_edges(ctx, n, *(torch.from_numpy(x.view(np.int32)).cuda() for x in (s, d)))
    fwh, fwc, bwh, bwc = G.to_host()
    want = O.tarjan(O.Graph(n, fwh, fwc, bwh, bwc))
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    for after in (0, 1):
        st = K.Stats()
        ctx.scc_device(n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options(aw_exact_after=after), st)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        got = st.as_dict()
        assert got["pivot"] == pivot and got["search_worklist"] == 1
        assert got["levels_bottom_up"] > 0 and got["heavy"]["cut_rows"] == len(hubs) and got["heavy"]["fixups"] > 0
