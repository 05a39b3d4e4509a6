"""Input checks at the edges of their vector loads: rows' arrays that start at
any 4-byte address, a fault at each place of a short array, and a valid call
on the same context afterwards (the launches behind a failed check leave the
graph alone)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _fails(ctx, G, arrays, out):
    import kaspan_b200 as K

    with pytest.raises(K.KspnError) as e:
        ctx.scc_device(G.n, G.m, *arrays, out, K.default_options())
    assert e.value.status == 2  # KSPN_ERR_INVALID_GRAPH


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n,draws", [(7, 3), (40, 21), (300, 1203)])
def test_faults_are_found_at_every_place(ctx, offset, n, draws):
    import torch

    import kaspan_b200 as K

    G = O.gnm(n, draws, 5)

    def rows(a):
        t = torch.zeros(len(a) + 8, dtype=torch.int32, device="cuda")
        t[offset: offset + len(a)] = torch.from_numpy(a.astype(np.uint32).view(np.int32)).cuda()
        return t[offset:]

    def heads(a):
        return torch.from_numpy(a.astype(np.uint64).view(np.int64)).cuda()

    arrays = [heads(G.fwh), rows(G.fwc), heads(G.bwh), rows(G.bwc)]
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    want = O.tarjan(G)
    places = sorted({0, 1, 2, 3, 4, G.m // 2, G.m - 5, G.m - 2, G.m - 1} & set(range(G.m)))
    for which in (1, 3):
        for p in places:
            keep = int(arrays[which][p])
            arrays[which][p] = n
            torch.cuda.synchronize()
            _fails(ctx, G, arrays, out)
            arrays[which][p] = keep
    for which in (0, 2):
        for p in (0, n // 2, n - 1, n):
            keep = int(arrays[which][p])
            arrays[which][p] = G.m + 1 if p < n else G.m - 1
            torch.cuda.synchronize()
            _fails(ctx, G, arrays, out)
            arrays[which][p] = keep
    torch.cuda.synchronize()
    ctx.scc_device(G.n, G.m, *arrays, out, K.default_options())
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
