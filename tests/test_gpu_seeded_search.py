"""Worklist phases that start from several vertices: long, thin graphs of
enough vertices for 8 to 73 start vertices, all of them in the pivot's SCC,
some of them, or none; and every take policy of the worklist.  Output
bit-identical to the oracle's Tarjan."""
from __future__ import annotations

import numpy as np
import pytest

import kaspan_b200 as K
import kaspan_b200.graphs as KG
import oracle as O

pytestmark = pytest.mark.gpu


N, SETS, SIZE = 100000, 12, 400


def build(kind):
    """A long cycle holding the pivot, and SETS small components whose
    vertices have the largest in * out of their 1024 ids: with N vertices, 24
    start vertices are tried, each the best of one such stretch, every other
    one of them in a set."""
    rng = np.random.default_rng(3)
    if kind == "grid":  # a sparse directed grid, many small components around a large one
        w = 300
        n = w * w + 7
        ids = np.arange(w * w).reshape(w, w)
        right, down = (ids[:, :-1].ravel(), ids[:, 1:].ravel()), (ids[:-1].ravel(), ids[1:].ravel())
        e = []
        for a, b in (right, down):
            r = rng.random(len(a))
            e += [(a[r < 0.62], b[r < 0.62]), (b[r > 0.38], a[r > 0.38])]
        perm = rng.permutation(n)
        s, d = (np.concatenate([x[i] for x in e]) for i in (0, 1))
        return n, perm[s].astype(np.uint32), perm[d].astype(np.uint32)
    blocks = -(-N // 1024)
    sets = [np.arange(i * blocks // SETS * 1024 + 100, i * blocks // SETS * 1024 + 100 + SIZE) for i in range(SETS)]
    if kind == "one_cycle":  # every start vertex in the pivot's SCC
        sets = []
    main = np.setdiff1d(np.arange(N), np.concatenate(sets) if sets else [])
    hub = main[50]
    e = [(main, np.roll(main, -1)), (np.full(30, hub), main[60:90]), (main[60:90], np.full(30, hub))]
    for c in sets:
        e += [(c, np.roll(c, -1)), (c, np.roll(c, -2))]
    into = lambda c, k: e.append((rng.choice(c, k), rng.choice(main, k)))  # noqa: E731
    out_of = lambda c, k: e.append((rng.choice(main, k), rng.choice(c, k)))  # noqa: E731
    for i, c in enumerate(sets):
        if kind == "upstream" or (kind in ("both", "through") and i % 2 == 0) or (kind == "some" and i == 5):
            into(c, 25)
        if kind == "downstream" or (kind in ("both", "through") and i % 2 == 1) or (kind == "some" and i == 8):
            out_of(c, 25)
        if kind == "some" and i not in (5, 8):  # the others belong to the pivot's SCC
            into(c, 3)
            out_of(c, 3)
    if kind == "through":  # a path and a cycle between start vertices before and after the pivot's SCC
        t = main[-1000:]
        e[0] = (main[:-1000], np.roll(main[:-1000], -1))
        e += [(t[:-1], t[1:]), (sets[0][:1], t[:1]), (t[-1:], sets[1][:1]), (t[300:301], t[200:201])]
    return N, np.concatenate([x[0] for x in e]).astype(np.uint32), np.concatenate([x[1] for x in e]).astype(np.uint32)


@pytest.mark.parametrize("after", [0, 1, 2000])
@pytest.mark.parametrize("kind", ["one_cycle", "upstream", "downstream", "both", "some", "through", "apart", "grid"])
def test_matches_tarjan(ctx, kind, after):
    import torch

    n, s, d = build(kind)
    G = KG.from_edges(ctx, n, torch.from_numpy(s.view(np.int32)).cuda(), torch.from_numpy(d.view(np.int32)).cuda())
    fwh, fwc, bwh, bwc = G.to_host()
    want = O.tarjan(O.Graph(n, fwh, fwc, bwh, bwc))
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    for pipeline in (K.PIPELINE_FAST, K.PIPELINE_FAST, K.PIPELINE_REFERENCE):  # the worklist must be left all zeros for the next call
        st = K.Stats()
        ctx.scc_device(n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options(pipeline=pipeline, aw_exact_after=after), st)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        if pipeline == K.PIPELINE_FAST:
            assert st.as_dict()["search_worklist"] == 1


@pytest.mark.parametrize("n", [16384, 32767, 32768, 65535, 300007])
def test_rgg_sizes(ctx, n):
    import torch

    G = KG.rgg(ctx, n, 5)
    fwh, fwc, bwh, bwc = G.to_host()
    want = O.tarjan(O.Graph(n, fwh, fwc[: max(G.m, 1)], bwh, bwc[: max(G.m, 1)]))
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    ctx.scc_device(n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options())
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
