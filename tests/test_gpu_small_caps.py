"""Caps on small graphs: a call with any of them runs the launches that count
against it, not the one-block decomposition, and is refused as on larger
graphs."""
import numpy as np
import pytest

import kaspan_b200 as K
import kaspan_b200.graphs as KG
import oracle as O

pytestmark = pytest.mark.gpu

SIZE, COUNT = 700, 4  # cycles too large for the residual step: label searches of 700 levels


@pytest.mark.parametrize("cap", ["max_levels", "max_label_iters"])
def test_caps_are_met(ctx, cap):
    import torch

    n = SIZE * COUNT
    s = np.arange(n)
    d = np.where(s % SIZE == SIZE - 1, s - SIZE + 1, s + 1)
    G = KG.from_edges(ctx, n, *(torch.from_numpy(x.astype(np.int32)).cuda() for x in (s, d)))
    fwh, fwc, bwh, bwc = G.to_host()
    want = O.tarjan(O.Graph(n, fwh, fwc, bwh, bwc))
    out = torch.empty(n, dtype=torch.int32, device="cuda")

    def run(**kw):
        st = K.Stats()
        ctx.scc_device(n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options(**kw), st)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        return st.as_dict()

    assert run()["kernel_launches"] == 1
    for limit in (1, 3):
        with pytest.raises(K.KspnError) as e:
            run(**{cap: limit})
        assert e.value.status == 4  # KSPN_ERR_TIMEOUT
    st = run(**{cap: n + 2})
    assert st["kernel_launches"] > 1 and st["label_calls"] >= 1
    assert run()["kernel_launches"] == 1
