"""The batched path's classes at their edges: graphs just inside and outside
the block sizes (512 or 2^15, and 2^18 vertices), the warp path (32 vertices), rows longer than a lane walks alone, degrees that need 32-bit counts,
and graphs whose rest after the first SCC is larger or smaller than it; each
against the oracle's Tarjan."""
import numpy as np
import pytest

import kaspan_b200.graphs as KG
import oracle as O

pytestmark = pytest.mark.gpu


def gnm(n, degree, seed):
    rng = np.random.default_rng(seed)
    m = int(n * degree)
    return n, rng.integers(0, n, m), rng.integers(0, n, m)


def hub(n, fan, seed):
    """A random graph with a hub that `fan` vertices point to and that points
    to `fan` others, and a chain into and out of it."""
    n, s, d = gnm(n, 1.3, seed)
    rng = np.random.default_rng(seed + 1)
    s = np.concatenate([s, rng.integers(1, n, fan), np.zeros(fan, np.int64), np.arange(n - 40, n - 1)])
    d = np.concatenate([d, np.zeros(fan, np.int64), rng.integers(1, n, fan), np.arange(n - 39, n)])
    return n, s, d


def two_parts(n, share, seed):
    """A dense part of `share` of the vertices, a sparse part, edges one way."""
    rng = np.random.default_rng(seed)
    k = int(n * share)
    s1, d1 = rng.integers(0, k, 4 * k), rng.integers(0, k, 4 * k)
    s2, d2 = rng.integers(k, n, int(1.2 * (n - k))), rng.integers(k, n, int(1.2 * (n - k)))
    s3, d3 = rng.integers(0, k, n // 8), rng.integers(k, n, n // 8)
    return n, np.concatenate([s1, s2, s3]), np.concatenate([d1, d2, d3])


def run(ctx, graphs):
    import torch

    sizes = np.array([g[0] for g in graphs], np.uint32)
    vo = np.concatenate([[0], np.cumsum(sizes, dtype=np.int64)])
    src = np.concatenate([g[1] + vo[i] for i, g in enumerate(graphs)])
    dst = np.concatenate([g[2] + vo[i] for i, g in enumerate(graphs)])
    N = int(vo[-1])
    G = KG.from_edges(ctx, N, torch.from_numpy(src.astype(np.int32)).cuda(), torch.from_numpy(dst.astype(np.int32)).cuda())
    ctx.synchronize()
    fwh, fwc = G.fwh.cpu().numpy().view(np.uint64), G.fwc.cpu().numpy().view(np.uint32)[: G.m].copy()
    want = O.tarjan(O.from_csr(N, fwh, fwc)).astype(np.int64) - np.repeat(vo[:-1], sizes)
    d_vo = torch.from_numpy(vo).cuda()
    for head, csr in ((G.fwh, G.fwc), (G.bwh, G.bwc)):
        ctx.batch_localize(len(graphs), N, d_vo, head, csr)
    out = torch.empty(N, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    st = ctx.scc_batched(len(graphs), N, d_vo, G.fwh, G.fwc, G.bwh, G.bwc, out)
    assert np.array_equal(out.cpu().numpy(), want)
    return st


@pytest.mark.parametrize("degree", [0.7, 1.0, 1.6, 4.0])
def test_class_edges(ctx, degree):
    sizes = [1, 31, 32, 33, 511, 512, 513, 600, 1023, 2049, 8191, 16384, 65535, 65536, 65537, 131071, 262143, 262144, 262145]
    run(ctx, [gnm(n, degree, 3 * n) for n in sizes])


@pytest.mark.parametrize("degree", [0.9, 1.6])
def test_classes_of_large_counts(ctx, degree):
    """More than two graphs per SM, where the larger block starts at 2^15
    vertices instead of 512; remainders around the first round's 64."""
    sizes = [32767, 32768, 32769, 511, 512, 513] + [20 + i % 60 for i in range(700)]
    run(ctx, [gnm(n, degree, 5 * n + i) for i, n in enumerate(sizes)])


@pytest.mark.parametrize("fan", [31, 33, 200, 254, 255, 256, 3000])
def test_hubs(ctx, fan):
    run(ctx, [hub(n, min(fan, n - 2), n + fan) for n in (700, 5000, 70000)])


@pytest.mark.parametrize("share", [0.05, 0.3, 0.5, 0.7, 0.95])
def test_rest_larger_and_smaller_than_the_scc(ctx, share):
    run(ctx, [two_parts(n, share, n) for n in (1500, 9001, 66000, 100003)])
