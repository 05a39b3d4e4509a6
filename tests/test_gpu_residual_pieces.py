"""The residual step at the edges of its piece classes: weakly connected
pieces of 1 to 513 vertices in shuffled ids, in every arrangement a piece is
handled by (closure of up to 32 vertices, shared-memory Tarjan of up to 512
vertices and 2048 internal edges, left over beyond that or with a row of
more than 2048 entries); ids against the oracle's Tarjan."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def piece(k, kind, rng):
    """Edges of one weakly connected piece on local ids 0 .. k - 1."""
    ids = np.arange(k)
    if kind == "cycle":
        e = [(ids, np.roll(ids, -1))]
    elif kind == "path":
        e = [(ids[:-1], ids[1:])]
    elif kind == "two_cycles":
        h = max(1, k // 2)
        e = [(ids[:h], np.roll(ids[:h], -1)), (ids[h:], np.roll(ids[h:], -1)), (ids[:1], ids[-1:])]
    else:  # random, connected through a path
        m = min(3 * k, 1500)
        e = [(rng.integers(0, k, m), rng.integers(0, k, m)), (np.minimum(ids[:-1], ids[1:]), np.maximum(ids[:-1], ids[1:]))]
    return np.concatenate([x[0] for x in e]), np.concatenate([x[1] for x in e])


def csr(n, s, d):
    order = np.lexsort((d, s))
    s, d = s[order], d[order]
    return np.searchsorted(s, np.arange(n + 1)).astype(np.uint64), d.astype(np.uint32)


@pytest.mark.parametrize("kind", ["cycle", "path", "two_cycles", "random"])
@pytest.mark.parametrize("sizes", [[1], [2], [31], [32], [33], [512], [513], [1, 2, 3, 5, 31, 32, 33, 64, 100, 511, 512, 513, 600], [4] * 3000, [33] * 200])
def test_pieces(ctx, kind, sizes):
    import torch

    rng = np.random.default_rng(len(sizes) + sum(sizes))
    n = sum(sizes) + 37
    perm = rng.permutation(n)  # the last 37 are decided already
    src, dst, at = [], [], 0
    for k in sizes:
        s, d = piece(k, kind, rng)
        src.append(perm[at + s]), dst.append(perm[at + d])
        at += k
    # edges through decided vertices join nothing
    src += [perm[rng.integers(0, at, 200)], perm[n - 37 + rng.integers(0, 37, 200)]]
    dst += [perm[n - 37 + rng.integers(0, 37, 200)], perm[rng.integers(0, at, 200)]]
    s, d = np.concatenate(src), np.concatenate(dst)
    live = np.ones(n, bool)
    live[perm[n - 37:]] = False
    keep = live[s] & live[d]
    want = O.tarjan(O.from_csr(n, *csr(n, s[keep], d[keep])))
    fwh, fwc = csr(n, s, d)
    bits = np.zeros((n + 63) // 64 * 64, np.uint8)
    bits[:n] = live
    und = torch.from_numpy(np.packbits(bits, bitorder="little").view(np.int64).copy()).cuda()
    ids = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    decided, left = ctx.residual(n, len(fwc), torch.from_numpy(fwh.view(np.int64)).cuda(), torch.from_numpy(fwc.view(np.int32)).cuda(), und, ids)
    big = [k for k in sizes if k > 512]
    assert decided == sum(sizes) - sum(big) and left == len(big)
    got = ids.cpu().numpy().view(np.uint32)
    after = np.unpackbits(und.cpu().numpy().view(np.uint8), bitorder="little")[:n].astype(bool)
    at = 0
    for k in sizes:
        p = perm[at: at + k]
        assert np.all(after[p] == (k > 512))
        assert np.array_equal(got[p], want[p] if k <= 512 else np.full(k, 0xFFFFFFFF, np.uint32))
        at += k
    assert np.all(got[perm[n - 37:]] == 0xFFFFFFFF)


@pytest.mark.parametrize("k,repeats,left", [(8, 255, 0), (8, 257, 1), (40, 51, 0), (40, 52, 1), (5, 2048, 1), (5, 2049, 1)])
def test_repeated_edges(ctx, k, repeats, left):
    """Cycles whose edges are repeated: left over from 2049 internal edges."""
    import torch

    s = np.repeat(np.arange(k), repeats)
    fwh, fwc = csr(k, s, (s + 1) % k)
    und = torch.tensor([(1 << k) - 1], dtype=torch.int64, device="cuda")
    ids = torch.full((k,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    decided, over = ctx.residual(k, len(fwc), torch.from_numpy(fwh.view(np.int64)).cuda(), torch.from_numpy(fwc.view(np.int32)).cuda(), und, ids)
    assert (decided, over) == (0 if left else k, left)
    assert np.all(ids.cpu().numpy() == (-1 if left else 0))
