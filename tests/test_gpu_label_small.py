"""Label searches over few undecided vertices (one block) beside the general
path: every pipeline that runs them, with leftovers just below and above the
one-block limits (32,768 vertices, 2^20 row entries, a row of 8192), deep
pieces, and the propagation cap; ids against the oracle's Tarjan."""
import numpy as np
import pytest

import kaspan_b200 as K
import kaspan_b200.graphs as KG
import oracle as O

pytestmark = pytest.mark.gpu

PIPELINES = [K.PIPELINE_FAST, K.PIPELINE_REFERENCE, K.PIPELINE_HPC_LIKE, K.PIPELINE_TRIM_EX]


def run(ctx, n, s, d, pipelines, **kw):
    import torch

    G = KG.from_edges(ctx, n, torch.from_numpy(s.astype(np.int32)).cuda(), torch.from_numpy(d.astype(np.int32)).cuda())
    fwh, fwc, bwh, bwc = G.to_host()
    want = O.tarjan(O.Graph(n, fwh, fwc, bwh, bwc))
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    for pipeline in pipelines:
        st = K.Stats()
        ctx.scc_device(G.n, G.m, G.fwh, G.fwc, G.bwh, G.bwc, out, K.default_options(pipeline=pipeline, **kw), st)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
    return st


def pieces(k, count, extra, seed, chain=True):
    """A dense core that the FW-BW takes, then `count` cycles of k vertices
    with chords, one feeding the next (pieces too large for the residual step)."""
    rng = np.random.default_rng(seed)
    core = 3 * k * count + 50
    n = core + k * count
    s, d = [rng.integers(0, core, 8 * core), np.arange(core)], [rng.integers(0, core, 8 * core), np.roll(np.arange(core), -1)]
    for i in range(count):
        ids = core + i * k + np.arange(k)
        s += [ids, rng.choice(ids, extra)]
        d += [np.roll(ids, -1), rng.choice(ids, extra)]
        if chain and i:
            s.append(ids[:1] - k)
            d.append(ids[5:6])
    return n, np.concatenate(s), np.concatenate(d)


@pytest.mark.parametrize("k,count,extra", [(600, 1, 0), (700, 3, 900), (3000, 2, 40), (32768, 1, 20000), (32769, 1, 20000), (30000, 1, 560000)])
def test_leftovers(ctx, k, count, extra):
    run(ctx, *pieces(k, count, extra, k + count), PIPELINES)


@pytest.mark.parametrize("fan", [8191, 8192, 8193])
def test_long_rows(ctx, fan):
    n, s, d = pieces(fan + 60, 1, 0, fan)
    hub = n - 1
    first = n - fan - 60
    run(ctx, n, np.concatenate([s, np.full(fan - 1, hub)]), np.concatenate([d, np.arange(first + 1, first + fan)]), PIPELINES[:2])


def test_near_critical_graph(ctx):
    rng = np.random.default_rng(1)
    n, m = 200003, 212000
    run(ctx, n, rng.integers(0, n, m), rng.integers(0, n, m), [K.PIPELINE_FAST, K.PIPELINE_HPC_LIKE])


def test_propagation_cap(ctx):
    n, s, d = pieces(2000, 1, 0, 4)
    with pytest.raises(K.KspnError) as e:
        run(ctx, n, s, d, [K.PIPELINE_FAST], max_label_iters=3)
    assert e.value.status == 4  # KSPN_ERR_TIMEOUT
    run(ctx, n, s, d, [K.PIPELINE_FAST])  # the context stays usable
