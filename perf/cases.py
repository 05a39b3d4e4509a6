"""Workloads whose speed matters to users of kaspan_b200.

Every case goes through the package's public entry points, on seeded
synthetic graphs of the shapes the benchmark and the tests use.  Kinds:

  scc    one decomposition of a graph resident on the GPU
         (Context.scc_device), default options unless the case says otherwise
  host   one decomposition of a forward CSR in pinned host memory: the
         drop-in call (Context.scc_host_ptr, kspn_scc); the upload, the
         transpose and the download of the ids are part of the call
  batch  thousands of small graphs in one call (Context.scc_batched)
  build  edge list -> CSR + transpose (Context.build_csr, Context.transpose)
  train  one training step of the pivot model: gradient and Adam
         (Context.mlp_gradient, Context.mlp_adam)
"""
from __future__ import annotations

import math

import numpy as np
import torch

import kaspan_b200 as K
import kaspan_b200.graphs as KG


def listed():
    return [
        # the smallest calls: a service that decomposes small dependency
        # graphs one by one; launches and synchronisations are the cost
        dict(name="scc_gnm_1000", kind="scc", graph="gnm", n=1000, degree=4.0),
        # directed G(n, m), n = 2^16, mean degree 8: the benchmark's small
        # configuration
        dict(name="scc_gnm_65536", kind="scc", graph="gnm", n=1 << 16, degree=8.0),
        # a sparse random graph near the giant-component threshold, odd n:
        # deep searches and long peeling chains
        dict(name="scc_gnm_sparse_3m", kind="scc", graph="gnm", n=3000017, degree=1.5),
        # R-MAT scale 24, the benchmark's single-graph configuration, called
        # as a new user calls it (the input is validated)
        dict(name="scc_rmat24", kind="scc", graph="rmat", scale=24, degree=16),
        # R-MAT scale 26 with the learned pivot, input trusted: the headline
        dict(name="scc_rmat26_learned", kind="scc", graph="rmat", scale=26, degree=16, validate=0, learned=1),
        # road-like graphs of high diameter and many small components: an odd
        # size, and the benchmark's configuration
        dict(name="scc_rgg_1m", kind="scc", graph="rgg", n=1000003),
        dict(name="scc_rgg_2e24", kind="scc", graph="rgg", n=1 << 24),
        # kaspan::scc's own phase order, with its label searches
        dict(name="scc_reference_rmat21", kind="scc", graph="rmat", scale=21, degree=16, pipeline="scc"),
        # the benchmark's batch: 4096 uneven graphs around the threshold
        dict(name="batch_4096", kind="batch", count=4096, log2_min=8, log2_max=18, deg_min=0.8, deg_max=6.0),
        # the drop-in call on a host graph without its transpose
        dict(name="host_rmat22", kind="host", graph="rmat", scale=22, degree=16),
        # input preparation: a raw edge list with duplicates and self-loops
        dict(name="build_rmat22", kind="build", graph="rmat", scale=22, degree=16),
        # one step of the pivot model's training (64 graphs x 1024 samples)
        dict(name="train_65536", kind="train", count=65536),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scc", "scc", "scc", "scc", "scc", "host", "batch", "build", "train"])
    if kind == "train":
        return dict(kind="train", count=_log_uniform(rng, 1000, 200000))
    if kind == "batch":
        lo = rng.choice([6, 8, 10])
        return dict(kind="batch", count=_log_uniform(rng, 16, 3000), log2_min=lo, log2_max=lo + rng.choice([3, 5, 8]),
                    deg_min=rng.choice([0.5, 0.8, 1.0]), deg_max=rng.choice([2.0, 4.0, 6.0]))
    graph = rng.choice(["gnm", "gnm", "rmat", "rgg"])
    top = 12_000_000 if kind == "scc" else 3_000_000
    case = dict(kind=kind, graph=graph)
    if graph == "rmat":
        case.update(scale=rng.randint(10, 24 if kind == "scc" else 21), degree=rng.choice([4, 8, 13, 16]))
    elif graph == "rgg":
        case.update(n=_log_uniform(rng, 700, top))
    else:
        case.update(n=_log_uniform(rng, 300, top), degree=round(rng.uniform(0.8, 10.0), 2))
    if kind == "scc":
        if rng.random() < 0.3:
            case["validate"] = 0
        if graph == "rmat" and rng.random() < 0.3:
            case["learned"] = 1
        if graph == "rmat" and case["scale"] <= 21 and rng.random() < 0.3:
            case["pipeline"] = rng.choice(["scc", "hpc_like", "ispan_like", "trim_ex"])
    return case


def _edges(ctx, case, seed):
    """Edge list (int32 tensors on the GPU) and the vertex count."""
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        draws = int(case["degree"]) << case["scale"]
    elif case["graph"] == "gnm":
        n = case["n"]
        draws = max(1, int(round(n * case["degree"])))
    else:
        n = case["n"]
        g, r2 = KG.rgg_params(n)
        draws = ctx.gen_rgg(n, seed, g, r2)
    src = torch.empty(max(draws, 1), dtype=torch.int32, device="cuda")
    dst = torch.empty(max(draws, 1), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    if case["graph"] == "rmat":
        ctx.gen_rmat(case["scale"], draws, seed, *KG.rmat_thresholds(0.57, 0.19, 0.19), True, src, dst)
    elif case["graph"] == "gnm":
        ctx.gen_gnm(n, draws, seed, src, dst)
    else:
        ctx.gen_rgg(n, seed, g, r2, src, dst, draws)
    return n, src[:draws], dst[:draws]


def _batch_shape(case):
    return K.batch_shape(case["count"], 1000, case["log2_min"], case["log2_max"], case["deg_min"], case["deg_max"])


def _batch(ctx, case, seed):
    """The uneven G(n, m) mix; the sizes belong to the case, the edges to the
    seed."""
    sizes, draws = _batch_shape(case)
    offsets = [np.concatenate([[0], np.cumsum(a, dtype=np.uint64)]).astype(np.int64) for a in (sizes, draws)]
    n, total = int(offsets[0][-1]), int(offsets[1][-1])
    vtx_off, draw_off = (torch.from_numpy(a).cuda() for a in offsets)
    src = torch.empty(max(total, 1), dtype=torch.int32, device="cuda")
    dst = torch.empty(max(total, 1), dtype=torch.int32, device="cuda")
    ctx.gen_batch(case["count"], seed, vtx_off, draw_off, src, dst)
    g = KG.from_edges(ctx, n, src[:total], dst[:total])
    for head, csr in ((g.fwh, g.fwc), (g.bwh, g.bwc)):
        ctx.batch_localize(case["count"], n, vtx_off, head, csr)
    return KG.DeviceBatch(case["count"], n, g.m, vtx_off, g.fwh, g.fwc, g.bwh, g.bwc, sizes)


def _model_inputs(case, seed):
    """Features, labels and a model in training as the pivot trainer meets
    them: log-degree features in [0, 1], shares, soft labels near 0 and 1."""
    rng = np.random.default_rng(seed)
    count = case["count"]
    x = rng.uniform(0.05, 0.8, (count, 8)).astype(np.float32)
    x[:, 4:6] = rng.integers(0, 65, (count, 2)).astype(np.float32) / 64
    x[:, 6] = rng.integers(0, 3, count).astype(np.float32) / 2
    y = np.where(rng.random(count) < 0.8, 1.0, rng.uniform(0.0, 0.1, count)).astype(np.float32)
    p = np.zeros(K.MLP_PARAMS, np.float32)
    p[:256] = rng.uniform(-1, 1, 256) / math.sqrt(8)
    p[256:288] = rng.uniform(-0.1, 0.1, 32)
    p[288:1312] = rng.uniform(-1, 1, 1024) / math.sqrt(32)
    p[1312:1344] = rng.uniform(-0.1, 0.1, 32)
    p[1344:1376] = rng.uniform(-1, 1, 32) / math.sqrt(32)
    m = rng.normal(0, 1e-3, K.MLP_PARAMS).astype(np.float32)
    v = rng.uniform(1e-6, 1e-5, K.MLP_PARAMS).astype(np.float32)
    return x, y, p, m, v


ADAM_LR, ADAM_STEP = 1e-2, 50


def prepare(case, seed):
    """What a user's program holds before the call, on the GPU (host cases:
    pinned host arrays)."""
    kind = case["kind"]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = K.Context(0, stream=stream)
        state = dict(kind=kind, stream=stream, ctx=ctx)
        if kind == "train":
            x, y, p, m, v = (torch.from_numpy(a).cuda() for a in _model_inputs(case, seed))
            state.update(x=x, y=y, p=p, m=m, v=v, grad=torch.empty_like(p), loss=torch.empty(1, device="cuda"))
            stream.synchronize()
            return state
        with K.Context(0, stream=stream) as maker:  # the generators' scratch goes with it
            if kind == "batch":
                b = _batch(maker, case, seed)
                state.update(graph=b, out=torch.empty(max(b.n, 1), dtype=torch.int32, device="cuda"))
            elif kind == "build":
                n, src, dst = _edges(maker, case, seed)
                state.update(n=n, src=src, dst=dst)
                for name, size, dtype in (("fwh", n + 1, torch.int64), ("bwh", n + 1, torch.int64), ("fwc", src.numel(), torch.int32), ("bwc", src.numel(), torch.int32)):
                    state[name] = torch.empty(size, dtype=dtype, device="cuda")
            else:
                n, src, dst = _edges(maker, case, seed)
                g = KG.from_edges(maker, n, src, dst)
                del src, dst
                if kind == "host":
                    state.update(n=g.n, m=g.m, fwh=g.fwh.cpu().pin_memory(), fwc=g.fwc.cpu().pin_memory(),
                                 out=torch.empty(max(g.n, 1), dtype=torch.int32).pin_memory())
                else:
                    opt = K.default_options(pipeline=K.PIPELINES[case["pipeline"]] if "pipeline" in case else K.PIPELINE_FAST,
                                            validate=case.get("validate", 1), learned_pivot=case.get("learned", 0))
                    if case.get("learned"):
                        ctx.set_pivot_model(K.default_pivot_model())
                    state.update(graph=g, opt=opt, out=torch.empty(max(g.n, 1), dtype=torch.int32, device="cuda"))
        stream.synchronize()
    return state


def run(state):
    kind, ctx = state["kind"], state["ctx"]
    if kind == "scc":
        g = state["graph"]
        ctx.scc_device(g.n, g.m, g.fwh, g.fwc, g.bwh, g.bwc, state["out"], state["opt"])
        return state["out"]
    if kind == "host":
        ctx.scc_host_ptr(state["n"], state["m"], state["fwh"], state["fwc"], None, None, state["out"])
        return state["out"]
    if kind == "batch":
        b = state["graph"]
        ctx.scc_batched(b.count, b.n, b.vtx_off, b.fwh, b.fwc, b.bwh, b.bwc, state["out"])
        return state["out"]
    with torch.cuda.stream(state["stream"]):
        if kind == "build":
            # build_csr consumes its edge list; this program keeps its own
            n, fwh, fwc, bwh, bwc = (state[k] for k in ("n", "fwh", "fwc", "bwh", "bwc"))
            src = state["src"].clone()
            m = ctx.build_csr(n, src.numel(), src, state["dst"].clone(), fwh, fwc)
            ctx.transpose(n, m, fwh, fwc, bwh, bwc)
            # the buffers hold the raw list's length: the end past m is cleared
            fwc[m:].zero_()
            bwc[m:].zero_()
            return fwh, fwc, bwh, bwc
        p, m, v = state["p"].clone(), state["m"].clone(), state["v"].clone()
        ctx.mlp_gradient(state["x"], state["y"], p, state["grad"], state["loss"])
        ctx.mlp_adam(p, state["grad"], m, v, ADAM_LR, ADAM_STEP)
        return dict(grad=state["grad"], loss=state["loss"], params=p, m=m, v=v)


def _shape(case):
    """(vertices, edges kept) of a graph case; the edges up to a few percent."""
    if case["graph"] == "rmat":
        return 1 << case["scale"], 0.98 * (int(case["degree"]) << case["scale"])
    if case["graph"] == "gnm":
        return case["n"], case["n"] * case["degree"]
    return case["n"], 4.0 * case["n"]


def work(case):
    """Bytes and operations of one pass.  A validated graph is read whole.  An
    input that is trusted needs both offset arrays and, to show which vertices
    are strongly connected, one neighbour per vertex and direction (a tree
    from the pivot and one to it)."""
    kind = case["kind"]
    if kind == "train":
        c = case["count"]
        macs = 8 * 32 + 32 * 32 + 32
        return dict(bytes=c * 36 + 8 * 4 * K.MLP_PARAMS, flops=6 * macs * c)
    if kind == "batch":
        sizes, draws = _batch_shape(case)
        n, m = float(sizes.sum(dtype=np.uint64)), float(draws.sum(dtype=np.uint64))
        return dict(bytes=2 * (8 * n + 4 * min(n, m)) + 4 * n, flops=0)
    n, m = _shape(case)
    csr = 8 * (n + 1) + 4 * m
    if kind == "host":
        return dict(bytes=csr + 4 * n, flops=0)
    if kind == "build":
        return dict(bytes=8 * m + 2 * csr, flops=0)
    if not case.get("validate", 1):
        csr = 8 * (n + 1) + 4 * min(n, m)
    return dict(bytes=2 * csr + 4 * n, flops=0)


def _bf16(a):
    return torch.from_numpy(a).bfloat16().double().numpy()


def exact(case, seed):
    """The training step in 64 bits (weights rounded to BF16 for the pass, as
    the model is defined); the other kinds return whole numbers."""
    if case["kind"] != "train":
        return None
    x, y, p, m, v = _model_inputs(case, seed)
    x, y, q = x.astype(np.float64), y.astype(np.float64), _bf16(p)
    w1, b1, w2, b2, w3, b3 = q[:256].reshape(32, 8), q[256:288], q[288:1312].reshape(32, 32), q[1312:1344], q[1344:1376], q[1376]
    a1 = x @ w1.T + b1
    h1 = np.maximum(a1, 0)
    a2 = h1 @ w2.T + b2
    h2 = np.maximum(a2, 0)
    z = h2 @ w3 + b3
    loss = np.mean(np.maximum(z, 0) - z * y + np.log1p(np.exp(-np.abs(z))))
    dz = (1 / (1 + np.exp(-z)) - y) / len(y)
    d2 = dz[:, None] * w3 * (a2 > 0)
    d1 = (d2 @ w2) * (a1 > 0)
    grad = np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ dz, [dz.sum()]])
    # the optimiser's constants are FP32 numbers
    beta1, beta2, eps, lr = (float(np.float32(c)) for c in (0.9, 0.999, 1e-8, ADAM_LR))
    m = beta1 * m.astype(np.float64) + (1 - beta1) * grad
    v = beta2 * v.astype(np.float64) + (1 - beta2) * grad * grad
    p = p.astype(np.float64) - lr * (m / (1 - beta1**ADAM_STEP)) / (np.sqrt(v / (1 - beta2**ADAM_STEP)) + eps)
    return dict(grad=grad, loss=np.array([loss]), params=p, m=m, v=v)
