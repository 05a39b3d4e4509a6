"""Input checks on every route a graph may take: the one-block decomposition's
own; the grid-wide launches' (vector loads over rows that start at any 4-byte
address, offsets checked by the trim pass), whose later launches -- the search,
and on sparse graphs the resume launch queued behind it -- must leave a faulty
graph alone; and a transpose built inside the call from offsets not checked
yet.  A valid call on the same context follows every fault."""
import numpy as np
import pytest

import kaspan_b200 as K
import oracle as O

pytestmark = pytest.mark.gpu

WIDE = 1 << 22  # a wait limit keeps small graphs on the grid-wide launches
ROUTES = {  # vertices, edge draws, wait limit
    "block 7": (7, 3, 0),
    "block 300": (300, 1203, 0),
    "grid 7": (7, 3, WIDE),
    "grid 40": (40, 21, WIDE),
    "grid 300": (300, 1203, WIDE),
    "queued resume": (20003, 80001, 0),
    "dense": (20003, 200001, 0),
}


def tensors(G, offset):
    import torch

    def rows(a):
        t = torch.zeros(G.m + 8, dtype=torch.int32, device="cuda")
        t[offset: offset + G.m] = torch.from_numpy(a[: G.m].astype(np.uint32).view(np.int32)).cuda()
        return t[offset:]

    def heads(a):
        return torch.from_numpy(a.astype(np.uint64).view(np.int64)).cuda()

    return [heads(G.fwh), rows(G.fwc), heads(G.bwh), rows(G.bwc)]


def faults(G, which):
    """(place, value): ids out of range at the edges of the vector loads;
    offsets that decrease, end early or late, or lie far past the rows."""
    n, m = G.n, G.m
    if which in (1, 3):
        return [(p, v) for p in sorted({0, 1, 2, 3, 4, m // 2, m - 5, m - 2, m - 1} & set(range(m))) for v in (n, -1)]
    return [(0, 1)] + [(p, v) for p in (n // 2, n - 1) for v in (m + 1, 1 << 40, -1)] + [(n, m - 1), (n, m + 1)]


def launches(ctx, G, arrays, out, want, limit):
    st = K.Stats()
    ctx.scc_device(G.n, G.m, *arrays, out, K.default_options(wait_limit=limit), st)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
    return st.as_dict()["kernel_launches"]


@pytest.mark.parametrize("own_transpose", [False, True])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("route", ROUTES)
def test_faults_are_refused(ctx, route, offset, own_transpose):
    import torch

    n, draws, limit = ROUTES[route]
    G = O.gnm(n, draws, 5)
    arrays = tensors(G, offset)
    used = arrays[:2] + ([None, None] if own_transpose else arrays[2:])
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    want = O.tarjan(G)
    torch.cuda.synchronize()
    before = launches(ctx, G, arrays, out, want, limit)
    assert (before == 1) == route.startswith("block")
    for which in (0, 1) if own_transpose else range(4):
        for place, value in faults(G, which):
            keep = int(arrays[which][place])
            arrays[which][place] = value
            torch.cuda.synchronize()
            with pytest.raises(K.KspnError) as e:
                ctx.scc_device(G.n, G.m, *used, out, K.default_options(wait_limit=limit))
            assert e.value.status == 2  # KSPN_ERR_INVALID_GRAPH
            arrays[which][place] = keep
        torch.cuda.synchronize()
        assert launches(ctx, G, used, out, want, limit) >= before


@pytest.mark.parametrize("pipeline", [K.PIPELINE_REFERENCE, K.PIPELINE_TRIM_EX])
def test_host_driven_pipelines(ctx, pipeline):
    import torch

    G = O.gnm(3001, 9001, 7)
    arrays = tensors(G, 3)
    out = torch.empty(G.n, dtype=torch.int32, device="cuda")
    for which in range(4):
        for place, value in faults(G, which):
            keep = int(arrays[which][place])
            arrays[which][place] = value
            torch.cuda.synchronize()
            with pytest.raises(K.KspnError) as e:
                ctx.scc_device(G.n, G.m, *arrays, out, K.default_options(pipeline=pipeline))
            assert e.value.status == 2
            arrays[which][place] = keep
    torch.cuda.synchronize()
    ctx.scc_device(G.n, G.m, *arrays, out, K.default_options(pipeline=pipeline))
    assert np.array_equal(out.cpu().numpy().view(np.uint32), O.tarjan(G))
