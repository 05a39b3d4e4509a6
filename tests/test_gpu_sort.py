"""Edge list -> CSR -> transpose on the GPU against numpy, at the sorts' tile
edges and for every number of passes (key widths of 1 to 26 bits)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RX_TILE, ET_TILE = 6144, 1024  # pairs per tile of the sort, edges per tile of the CSR pass


def check(ctx, n, src, dst):
    import torch

    s, d = (torch.from_numpy(a.astype(np.int32)).cuda() for a in (src, dst))
    fwh, bwh = (torch.full((n + 1,), -1, dtype=torch.int64, device="cuda") for _ in range(2))
    fwc, bwc = (torch.full((max(len(src), 1),), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    m = ctx.build_csr(n, len(src), s, d, fwh, fwc)
    pairs = np.unique((src.astype(np.int64) << 32) | dst) if len(src) else np.zeros(0, np.int64)
    u, v = pairs >> 32, pairs & 0xFFFFFFFF
    u, v = u[u != v], v[u != v]
    assert m == len(u)
    ids = np.arange(n + 1)
    assert np.array_equal(fwh.cpu().numpy(), np.searchsorted(u, ids))
    assert np.array_equal(fwc[:m].cpu().numpy(), v)
    ctx.transpose(n, m, fwh, fwc, bwh, bwc)
    ctx.synchronize()
    order = np.argsort(v, kind="stable")
    assert np.array_equal(bwh.cpu().numpy(), np.searchsorted(v[order], ids))
    assert np.array_equal(bwc[:m].cpu().numpy(), u[order])


@pytest.mark.parametrize("m", [0, 1, 2, 31, 33, ET_TILE - 1, ET_TILE, ET_TILE + 1, RX_TILE - 1, RX_TILE, RX_TILE + 1, 2 * RX_TILE, 40 * RX_TILE + 17, 700001])
@pytest.mark.parametrize("bits", [1, 7, 8, 9, 16, 17, 24, 25, 26])
def test_tile_edges_and_passes(ctx, m, bits):
    rng = np.random.default_rng(m * 64 + bits)
    n = (1 << bits) - int(rng.integers(0, 1 << max(0, bits - 2)))
    check(ctx, n, rng.integers(0, n, m), rng.integers(0, n, m))


@pytest.mark.parametrize("kind", ["one_row", "one_column", "loops", "repeats", "last_ids"])
def test_skewed_edges(ctx, kind):
    rng = np.random.default_rng(7)
    n, m = 70001, 200003
    src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
    if kind == "one_row":
        src[:] = n - 1
    elif kind == "one_column":
        dst[:] = 0
    elif kind == "loops":
        dst[::2] = src[::2]
    elif kind == "repeats":
        src, dst = src % 13, dst % 11
    else:
        src, dst = n - 1 - src % 5, n - 1 - dst % 7
    check(ctx, n, src, dst)
