"""Graphs decomposed in one block (kernel_launches == 1) beside the grid-wide
path, up to both sides of the shared-memory limit: ids against the oracle's
Tarjan, the per-phase counts against the grid-wide path's."""
import numpy as np
import pytest

import kaspan_b200 as K
import oracle as O

pytestmark = pytest.mark.gpu


def csr(n, s, d):
    """Rows as given: self-loops and repeats stay."""
    import torch

    def rows(a, b):
        order = np.lexsort((b, a))
        return np.concatenate([[0], np.cumsum(np.bincount(a, minlength=n))]).astype(np.uint64), b[order].astype(np.uint32)

    (fh, fc), (bh, bc) = rows(s, d), rows(d, s)
    pad = lambda a: np.concatenate([a, np.zeros(1, a.dtype)])  # no array is empty
    dev = [torch.from_numpy(pad(a).view(np.int64 if a.dtype == np.uint64 else np.int32)).cuda() for a in (fh, fc, bh, bc)]
    return O.Graph(n, fh, fc, bh, bc), dev


def random_edges(n, m, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(0, n, m), rng.integers(0, n, m)


def chain_of_cycles(k, count, seed):
    n = k * count
    name = np.random.default_rng(seed).permutation(n)
    i = np.arange(n)
    nxt = np.where(i % k == k - 1, i - k + 1, i + 1)
    s, d = np.concatenate([i, i[k - 1:-1:k]]), np.concatenate([nxt, i[k::k]])
    return n, name[s], name[d]


def case(kind):
    if kind == "empty rows":
        return 70, np.array([], dtype=np.int64), np.array([], dtype=np.int64)
    if kind == "one vertex":
        return 1, np.array([0]), np.array([0])
    if kind == "loops and repeats":
        s, d = random_edges(33, 60, 1)
        return 33, np.concatenate([s, s, np.arange(0, 33, 2)]), np.concatenate([d, d, np.arange(0, 33, 2)])
    if kind == "hub":
        i = np.arange(1, 6001)
        return 6001, np.concatenate([np.zeros(6000, int), i[::2], i[:-1:3]]), np.concatenate([i, np.zeros(3000, int), i[1::3]])
    if kind == "path":
        return 9000, np.arange(8999), np.arange(1, 9000)
    if kind == "cycle":
        return 4097, np.arange(4097), np.roll(np.arange(4097), -1)
    if kind == "chain of 3-cycles":
        return chain_of_cycles(3, 1200, 3)
    if kind == "chain of 1200-cycles":
        return chain_of_cycles(1200, 6, 4)
    n, m = kind
    return (n, *random_edges(n, m, n + m))


@pytest.mark.parametrize("kind", ["empty rows", "one vertex", "loops and repeats", "hub", "path", "cycle", "chain of 3-cycles", "chain of 1200-cycles",
                                  (31, 60), (32, 64), (65, 90), (1000, 1100), (1025, 4000), (3000, 57000), (8000, 32000), (15000, 10000), (9000, 30000), (1000, 65535), (1000, 65536)])
def test_ids_and_counts(ctx, kind):
    import torch

    n, s, d = case(kind)
    G, dev = csr(n, s, d)
    want = O.tarjan(G)
    out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    res = {}
    # the wait limit is a hook of the grid-wide launches: it keeps the call on them
    for limit in (0, 1 << 22):
        st = K.Stats()
        out.fill_(-1)
        torch.cuda.synchronize()
        ctx.scc_device(n, len(s), *dev, out, K.default_options(wait_limit=limit), st)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)
        res[limit] = st.as_dict()
    few, wide = res.values()
    fits = 4 * len(s) + 12.5 * n < 226 * 1024 - 64 and len(s) <= 0xFFFF
    assert (few["kernel_launches"] == 1) == fits and wide["kernel_launches"] > 1
    assert few["pivot"] == wide["pivot"]
    for phase in ("trim_first", "fwbw", "trim"):
        assert few["decided"][phase] == wide["decided"][phase]


def test_unchecked_view_takes_the_wide_path(ctx):
    """Offsets that start past zero are refused when checked and work
    unchecked, as on larger graphs."""
    import torch

    n, s, d = case((1000, 4000))
    G, dev = csr(n, s, d)
    heads = [dev[0] + 8, dev[2] + 8]
    rows = [torch.cat([torch.zeros(8, dtype=torch.int32, device="cuda"), dev[i]]) for i in (1, 3)]
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    args = (n, len(s), heads[0], rows[0], heads[1], rows[1], out)
    with pytest.raises(K.KspnError):
        ctx.scc_device(*args, K.default_options())
    ctx.scc_device(*args, K.default_options(validate=0))
    assert np.array_equal(out.cpu().numpy().view(np.uint32), O.tarjan(G))
