"""Performance cases: the work a user of the library has it do, through the
public entry points of evoc_gb300.py.

A case is a dict of plain values; its "kind" names the call:

    evoc_host    evoc()'s pipeline on host arrays: fuzzy set, label-propagation
                 init, embedding, MST (the Rust caller's buffers)
    evoc_device  the same pipeline with kNN lists, points and results on the GPU
    graph        the fuzzy simplicial set of host kNN lists, exported into kept CSR buffers
    layout       fuzzy set, plan and epochs of device kNN lists
    restart      the epoch loop of a kept plan, from a given initial embedding
    batch        many problems: one block-diagonal fuzzy set, then embed_blocks
    lp_init      the label-propagation initialisation of a device graph and points
    mst          the mutual-reachability MST of a device layout
    predict      the warm-start network's prediction for device points
    gradients    its loss and gradients for a host batch
    fit          its training on device layouts

Points are seeded mixtures on the unit sphere (Zipf cluster sizes, child
clusters around parents, uniform noise), as in workloads.py; the kNN search is
exact inside cells of neighbouring clusters plus a sample of the other points,
so the graphs have the hubs and the uneven in-degrees of an ANN result.
"""
from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parents[1] / "evoc-rs_gb300"


@functools.lru_cache(maxsize=1)
def _lib():
    # the tree that is imported from is the working folder's, where there is one
    local = Path.cwd() / "evoc-rs_gb300"
    for p in (str(local), str(_PKG)):
        if Path(p).is_dir():
            sys.path.insert(0, p)
            break
    import evoc_gb300
    return evoc_gb300


@functools.lru_cache(maxsize=1)
def _ctx():
    """One context per process, as a user's program keeps one."""
    return _lib().Context(0)


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one of the smallest problems of a batch, alone, all on host arrays: launches and
        # synchronisations decide
        {"name": "evoc_host_2k", "kind": "evoc_host", "n": 2003, "d": 384, "k": 15, "dim": 4},
        # the ordinary call: the 200k x 512 configuration, everything device-resident
        {"name": "evoc_device_200k", "kind": "evoc_device", "n": 200_000, "d": 512, "k": 15,
         "dim": 8},
        # a caller that only wants the fuzzy graph (coo_to_adjacency_list on the host)
        {"name": "graph_50k", "kind": "graph", "n": 49_999, "d": 128, "k": 15,
         "symmetrise": True},
        # the headline configuration: 2M points, k 30, dim 8, 50 epochs from random
        {"name": "layout_2m", "kind": "layout", "n": 2_000_000, "d": 64, "k": 30, "dim": 8,
         "epochs": 50, "rate": 1.0},
        # more epochs and negatives than the default, the widest embedding
        {"name": "layout_61k_e100", "kind": "layout", "n": 61_003, "d": 64, "k": 20, "dim": 16,
         "epochs": 100, "rate": 2.0},
        # several runs of one kept plan (other starting layouts, the warm start)
        {"name": "restart_500k", "kind": "restart", "n": 500_000, "d": 64, "k": 15, "dim": 8,
         "epochs": 50},
        # many problems of uneven size in one call
        {"name": "batch_48", "kind": "batch", "problems": 48, "lo": 2000, "hi": 40_000, "d": 64,
         "k": 15, "dim": 4},
        # the initialisation alone at the largest size, with its 768-d points
        {"name": "lp_init_2m", "kind": "lp_init", "n": 2_000_000, "d": 768, "k": 30, "dim": 8},
        # the clustering stage's tree at 1M points
        {"name": "mst_1m", "kind": "mst", "n": 1_000_000, "dim": 8, "min_samples": 5},
        # the warm start's network: prediction for a whole data set, a gradient, a training run
        {"name": "predict_1m", "kind": "predict", "n": 1_000_000, "d": 768, "hidden": 512,
         "dim": 8},
        {"name": "gradients_8k", "kind": "gradients", "n": 8192, "d": 768, "hidden": 512,
         "dim": 8},
        {"name": "fit_200", "kind": "fit", "n": 60_000, "instances": 4, "d": 768, "hidden": 512,
         "dim": 8, "batch": 8192, "steps": 200},
    ]


def _log_int(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, v))


def draw(rng):
    kind = rng.choice(["evoc_host", "evoc_device", "graph", "layout", "layout", "restart", "batch",
                       "lp_init", "mst", "predict", "gradients", "fit"])
    k = rng.choice([10, 15, 15, 20, 30])
    dim = rng.choice([2, 3, 4, 5, 8, 8, 16])
    if kind == "evoc_host":
        return {"kind": kind, "n": _log_int(rng, 1500, 40_000), "d": rng.choice([50, 128, 384]),
                "k": k, "dim": dim}
    if kind == "evoc_device":
        return {"kind": kind, "n": _log_int(rng, 5000, 400_000), "d": rng.choice([128, 300, 512]),
                "k": k, "dim": dim}
    if kind == "graph":
        return {"kind": kind, "n": _log_int(rng, 1500, 200_000), "d": 64,
                "k": rng.choice([5, 10, 15, 30, 50]), "symmetrise": rng.random() < 0.75}
    if kind == "layout":
        n = _log_int(rng, 2000, 2_000_000)
        epochs = rng.choice([30, 50, 50, 50, 100]) if n < 300_000 else 50
        rate = rng.choice([1.0, 1.0, 1.0, 2.0, 5.0]) if n < 300_000 else 1.0
        return {"kind": kind, "n": n, "d": 64, "k": k, "dim": dim if n < 1_000_000 else 8,
                "epochs": epochs, "rate": rate}
    if kind == "restart":
        return {"kind": kind, "n": _log_int(rng, 2000, 1_000_000), "d": 64, "k": k, "dim": dim,
                "epochs": rng.choice([12, 20, 50])}
    if kind == "batch":
        lo = _log_int(rng, 1500, 4000)
        return {"kind": kind, "problems": rng.randrange(3, 49), "lo": lo,
                "hi": lo * rng.randrange(2, 10), "d": 64, "k": 15, "dim": rng.choice([2, 4, 8])}
    if kind == "lp_init":
        return {"kind": kind, "n": _log_int(rng, 5000, 1_500_000), "d": rng.choice([96, 384, 768]),
                "k": k, "dim": dim}
    if kind == "mst":
        return {"kind": kind, "n": _log_int(rng, 2000, 1_000_000), "dim": dim,
                "min_samples": rng.choice([1, 5, 5, 10, 25])}
    if kind == "predict":
        return {"kind": kind, "n": _log_int(rng, 300, 1_000_000), "d": rng.choice([256, 384, 768]),
                "hidden": rng.choice([256, 512]), "dim": dim}
    if kind == "gradients":
        return {"kind": kind, "n": _log_int(rng, 500, 20_000), "d": rng.choice([256, 384, 768]),
                "hidden": rng.choice([256, 512]), "dim": dim}
    return {"kind": kind, "n": _log_int(rng, 5000, 60_000), "instances": rng.randrange(1, 5),
            "d": rng.choice([256, 384, 768]), "hidden": rng.choice([256, 512]), "dim": dim,
            "batch": rng.choice([1024, 4096, 8192]), "steps": rng.randrange(30, 200)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _unit(x):
    return x / x.norm(dim=1, keepdim=True)


def _points(n, d, g):
    """n unit rows in cluster order (noise last): child clusters at 0.2 rad around
    parents, Zipf(1.0) sizes, 5% uniform noise, spread 0.42 in norm."""
    parents = max(2, min(50, n // 1500))
    nc = parents * 10
    noise = n // 20
    w = 1.0 / np.arange(1, nc + 1)
    sizes = np.floor(w / w.sum() * (n - noise)).astype(np.int64)
    sizes[0] += (n - noise) - sizes.sum()
    pc = _unit(torch.randn(parents, d, generator=g, device="cuda"))
    u = torch.randn(nc, d, generator=g, device="cuda")
    pr = pc.repeat_interleave(10, 0)
    u = _unit(u - (u * pr).sum(1, keepdim=True) * pr)
    child = math.cos(0.2) * pr + math.sin(0.2) * u
    child = child[torch.randperm(nc, generator=g, device="cuda")]
    lab = torch.repeat_interleave(torch.arange(nc, device="cuda"),
                                  torch.from_numpy(sizes).cuda(), output_size=n - noise)
    x = torch.randn(n, d, generator=g, device="cuda")
    x[:n - noise].mul_(0.42 / math.sqrt(d)).add_(child[lab])
    return x.div_(x.norm(dim=1, keepdim=True))


def _knn(n, d, k, g, keep_points):
    """Cosine kNN lists (int32 idx, f32 dist, n x k, nearest first, self removed) of
    shuffled points, and the points where they are kept."""
    x = _points(n, d, g)
    cell = 4096 if n <= 500_000 else 2048
    idx = torch.empty(n, k, dtype=torch.int64, device="cuda")
    dist = torch.empty(n, k, dtype=torch.float32, device="cuda")
    mark = torch.randperm(n, generator=g, device="cuda")[:512]
    xm = x[mark]
    cuts = list(range(0, max(1, n - cell // 2), cell)) + [n]
    for a, b in zip(cuts[:-1], cuts[1:]):
        sim = x[a:b] @ torch.cat([x[a:b], xm]).T
        m = b - a
        sim[:, :m].fill_diagonal_(-2.0)
        sim[:, m:].masked_fill_(((mark >= a) & (mark < b))[None, :], -2.0)
        top = torch.topk(sim, k, dim=1)
        idx[a:b] = torch.where(top.indices < m, top.indices + a,
                               mark[(top.indices - m).clamp_min(0)])
        dist[a:b] = (1.0 - top.values).clamp_min(0.0)
    new = torch.randperm(n, generator=g, device="cuda")  # ordered row -> shuffled id
    old = torch.argsort(new)
    out_i = new[idx][old].to(torch.int32).contiguous()
    out_d = dist[old].contiguous()
    return out_i, out_d, (x[old].contiguous() if keep_points else None)


def _layout_points(n, dim, g):
    """A layout as the embedding leaves it: compact clusters of uneven size and width
    on wider groups, a few stray points."""
    groups, per = 40, 8
    nc = groups * per
    w = 1.0 / torch.arange(1, nc + 1, device="cuda", dtype=torch.float64)
    lab = torch.multinomial(w, n, replacement=True, generator=g)
    top = 6.0 * torch.randn(groups, dim, generator=g, device="cuda")
    c = top.repeat_interleave(per, 0) + 0.8 * torch.randn(nc, dim, generator=g, device="cuda")
    c = c[torch.randperm(nc, generator=g, device="cuda")]
    width = torch.exp(torch.randn(nc, dim, generator=g, device="cuda") * 0.5) * 0.15
    x = c[lab] + width[lab] * torch.randn(n, dim, generator=g, device="cuda")
    stray = torch.rand(n, generator=g, device="cuda") < 0.02
    x = torch.where(stray[:, None], 7.0 * torch.randn(n, dim, generator=g, device="cuda"), x)
    return x.contiguous()


def _sizes(case):
    """Point counts of a batch's problems: log-uniform, in mixed order."""
    m = case["problems"]
    at = (np.arange(m) * 7919 % m + 0.5) / m if m % 7919 else (np.arange(m) + 0.5) / m
    return [int(case["lo"] * (case["hi"] / case["lo"]) ** q) for q in at]


def _net_inputs(case, seed):
    """Unit points as BF16-representable f32, and a layout-like target."""
    g = _gen(seed)
    n = case["n"]
    x = torch.randn(n, case["d"], generator=g, device="cuda") / math.sqrt(case["d"])
    centres = torch.randn(32, case["d"], generator=g, device="cuda") / math.sqrt(case["d"])
    lab = torch.randint(0, 32, (n,), generator=g, device="cuda")
    x = _unit(0.5 * x + centres[lab])
    t = torch.randn(32, case["dim"], generator=g, device="cuda")[lab]
    t = t + 0.1 * torch.randn(n, case["dim"], generator=g, device="cuda")
    return x.to(torch.bfloat16).contiguous(), t.contiguous()


def _weights(case, seed):
    """Packed W1, b1, W2, b2, W3, b3 of a network (uniform, 1 / sqrt(fan in))."""
    rng = np.random.default_rng(seed + 17)
    i, h, o = case["d"], case["hidden"], case["dim"]
    out = []
    for count, fan in ((h * i, i), (h, i), (h * h, h), (h, h), (o * h, h), (o, h)):
        out.append(rng.uniform(-1.0, 1.0, count) / math.sqrt(fan))
    return np.concatenate(out).astype(np.float32)


def prepare(case, seed):
    E, ctx, kind = _lib(), _ctx(), case["kind"]
    g = _gen(seed)
    st = {"case": case, "E": E, "ctx": ctx, "seed": int(seed) + 42}
    n, k, dim = case.get("n"), case.get("k"), case.get("dim")

    def empty(*shape, dtype=torch.float32):
        return torch.empty(*shape, dtype=dtype, device="cuda")

    if kind in ("evoc_host", "graph"):
        idx, dist, x = _knn(n, case["d"], k, g, kind == "evoc_host")
        st["idx"] = idx.cpu().numpy().astype(np.uint32)
        st["dist"] = dist.cpu().numpy()
        st["x"] = None if x is None else x.cpu().numpy()
        if kind == "graph":  # a caller's CSR buffers, kept and large enough for any union
            st["indptr"] = np.zeros(n + 1, np.int64)
            st["indices"] = np.zeros(2 * n * k, np.uint32)
            st["weights"] = np.zeros(2 * n * k, np.float32)
    elif kind in ("evoc_device", "layout"):
        st["idx"], st["dist"], st["x"] = _knn(n, case["d"], k, g, kind == "evoc_device")
        st["out"] = empty(n, dim)
        if kind == "layout":
            st["sigma"], st["rho"] = empty(n), empty(n)
        else:
            st["init"] = empty(n, dim)
            st["u"], st["v"], st["w"] = (empty(n - 1, dtype=torch.int64),
                                         empty(n - 1, dtype=torch.int64), empty(n - 1))
    elif kind in ("restart", "lp_init"):
        idx, dist, st["x"] = _knn(n, case["d"], k, g, kind == "lp_init")
        st["out"] = empty(n, dim)
        torch.cuda.synchronize()
        graph = ctx.fuzzy_set_device(idx.data_ptr(), dist.data_ptr(), n, k, float(k), True)
        if kind == "restart":
            st["plan"] = ctx.plan(graph, dim, E.EvocEmbeddingParams(n_epochs=case["epochs"]),
                                  seed=st["seed"])
            st["init"] = 0.1 * _layout_points(n, dim, g)
            graph.free()
        else:
            st["graph"] = graph
    elif kind == "batch":
        st["sizes"] = _sizes(case)
        st["knn"] = []
        for m in st["sizes"]:
            idx, dist, _ = _knn(m, case["d"], k, g, False)
            st["knn"].append((idx.cpu().numpy().astype(np.uint32), dist.cpu().numpy()))
    elif kind == "mst":
        st["x"] = _layout_points(n, dim, g)
        st["u"], st["v"], st["w"] = (empty(n - 1, dtype=torch.int64),
                                     empty(n - 1, dtype=torch.int64), empty(n - 1))
    elif kind == "predict":
        st["net"] = ctx.mlp(case["d"], case["hidden"], dim, seed=st["seed"])
        st["net"].set_params(_weights(case, seed))
        st["x"], _ = _net_inputs(case, seed)
        st["out"] = empty(n, dim)
    elif kind == "gradients":
        st["net"] = ctx.mlp(case["d"], case["hidden"], dim, seed=st["seed"])
        st["net"].set_params(_weights(case, seed))
        x, t = _net_inputs(case, seed)
        st["x"], st["t"] = x.float().cpu().numpy(), t.cpu().numpy()
    elif kind == "fit":
        st["net"] = ctx.mlp(case["d"], case["hidden"], dim, seed=st["seed"])
        st["weights"] = _weights(case, seed)
        st["inst"] = [_net_inputs(case, seed + 1000 * q) for q in range(case["instances"])]
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    case, ctx, E = st["case"], st["ctx"], st["E"]
    kind = case["kind"]
    n, k, dim = case.get("n"), case.get("k"), case.get("dim")
    if kind == "evoc_host":
        graph = E.build_fuzzy_simplicial_set(ctx, st["idx"], st["dist"], float(k), True)
        init = ctx.label_propagation_init(graph, dim, st["x"], seed=st["seed"])
        emb = E.evoc_embedding(ctx, graph, dim, None, init, seed=st["seed"])
        u, v, w = ctx.build_mst(emb, 5)
        graph.free()
        return {"init": init, "embedding": emb, "u": u, "v": v, "w": w}
    if kind == "evoc_device":
        graph = ctx.fuzzy_set_device(st["idx"].data_ptr(), st["dist"].data_ptr(), n, k, float(k),
                                     True)
        ctx.label_propagation_init_device(graph, dim, st["x"].data_ptr(), case["d"], st["seed"],
                                          st["init"].data_ptr())
        plan = ctx.plan(graph, dim, seed=st["seed"])
        plan.run_device(st["init"].data_ptr(), st["out"].data_ptr())
        plan.free()
        m = ctx.build_mst_device(st["out"].data_ptr(), n, dim, 5, st["u"].data_ptr(),
                                 st["v"].data_ptr(), st["w"].data_ptr())
        nnz = graph.nnz
        graph.free()
        return {"nnz": nnz, "init": st["init"], "embedding": st["out"], "edges": m, "u": st["u"],
                "v": st["v"], "w": st["w"]}
    if kind == "graph":
        graph = E.build_fuzzy_simplicial_set(ctx, st["idx"], st["dist"], float(k),
                                             case["symmetrise"])
        nnz = graph.nnz
        ctx._check(ctx.lib.evoc_graph_export(graph.handle, st["indptr"].ctypes.data,
                                             st["indices"].ctypes.data, st["weights"].ctypes.data))
        graph.free()
        return {"nnz": nnz, "indptr": st["indptr"], "indices": st["indices"],
                "weights": st["weights"]}
    if kind == "layout":
        graph = ctx.fuzzy_set_device(st["idx"].data_ptr(), st["dist"].data_ptr(), n, k, float(k),
                                     True, st["sigma"].data_ptr(), st["rho"].data_ptr())
        params = E.EvocEmbeddingParams(n_epochs=case["epochs"], negative_sample_rate=case["rate"])
        plan = ctx.plan(graph, dim, params, seed=st["seed"])
        plan.run_device(None, st["out"].data_ptr())
        plan.free()
        nnz = graph.nnz
        graph.free()
        return {"nnz": nnz, "sigma": st["sigma"], "rho": st["rho"], "embedding": st["out"]}
    if kind == "restart":
        st["plan"].run_device(st["init"].data_ptr(), st["out"].data_ptr())
        return {"embedding": st["out"]}
    if kind == "batch":
        graph = ctx.fuzzy_set_batched(st["knn"], float(k), True)
        outs = ctx.embed_blocks(graph, st["sizes"], dim, seeds=[st["seed"]] * len(st["sizes"]))
        graph.free()
        return {"embeddings": outs}
    if kind == "lp_init":
        ctx.label_propagation_init_device(st["graph"], dim, st["x"].data_ptr(), case["d"],
                                          st["seed"], st["out"].data_ptr())
        return {"init": st["out"]}
    if kind == "mst":
        m = ctx.build_mst_device(st["x"].data_ptr(), n, dim, case["min_samples"],
                                 st["u"].data_ptr(), st["v"].data_ptr(), st["w"].data_ptr())
        return {"edges": m, "u": st["u"], "v": st["v"], "w": st["w"]}
    if kind == "predict":
        st["net"].predict_device(st["x"].data_ptr(), n, st["out"].data_ptr())
        return {"y": st["out"]}
    if kind == "gradients":
        loss, grad = st["net"].gradients(st["x"], st["t"])
        return {"loss": loss, "grad": grad}
    if kind == "fit":
        net, inst = st["net"], st["inst"]
        net.set_params(st["weights"])
        hist = net.fit_device([x.data_ptr() for x, _ in inst], [t.data_ptr() for _, t in inst],
                              [n] * len(inst),
                              E.MlpTrainParams(steps=case["steps"], batch=case["batch"]))
        return {"loss": hist, "params": net.get_params()}
    raise ValueError(kind)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _graph_flops(n, k):
    # about 27 bisection steps of k exponentials (an exponential: about 20 operations)
    return n * k * 28 * 20.0


def _epoch_flops(n, k, dim, epochs, rate):
    # about n k 0.9 undirected edges, 16% of them fired in an epoch, each from both ends,
    # each end with `rate` negatives; then Adam on every node
    fired = 0.16 * 0.9 * n * k
    return epochs * (fired * (2.0 + rate) * (5 * dim + 10) + n * dim * 12.0)


def work(case):
    kind = case["kind"]
    n, k, dim, d = case.get("n"), case.get("k"), case.get("dim"), case.get("d")
    if kind == "batch":
        n = sum(_sizes(case))
    if kind in ("evoc_host", "evoc_device"):
        return {"bytes": 8.0 * n * k + 4.0 * n * d + 8.0 * n * dim + 20.0 * n,
                "flops": _graph_flops(n, k) + _epoch_flops(n, k, dim, 50, 1.0) + 2.0 * n * d +
                n * math.log2(n) * 4 * dim}
    if kind == "graph":
        ratio = 1.75 if case["symmetrise"] else 1.0
        return {"bytes": 8.0 * n * k + 8.0 * n + 8.0 * ratio * n * k, "flops": _graph_flops(n, k)}
    if kind == "layout":
        return {"bytes": 8.0 * n * k + 8.0 * n + 4.0 * n * dim,
                "flops": _graph_flops(n, k) +
                _epoch_flops(n, k, dim, case["epochs"], case["rate"])}
    if kind == "restart":
        return {"bytes": 8.0 * n * dim + 1.75 * 8.0 * n * k,
                "flops": _epoch_flops(n, k, dim, case["epochs"], 1.0)}
    if kind == "batch":
        return {"bytes": 8.0 * n * k + 4.0 * n * dim,
                "flops": _graph_flops(n, k) + _epoch_flops(n, k, dim, 50, 1.0)}
    if kind == "lp_init":
        return {"bytes": 4.0 * n * d + 1.75 * 8.0 * n * k + 4.0 * n * dim,
                "flops": 2.0 * n * d + 1.75 * n * k * (4.0 + 2.0 * dim)}
    if kind == "mst":
        return {"bytes": 4.0 * n * dim + 20.0 * n,
                "flops": n * math.log2(n) * 4.0 * dim + n * case["min_samples"] * 3.0 * dim}
    per_row = d * case["hidden"] + case["hidden"] ** 2 + case["hidden"] * dim
    params = per_row + 2 * case["hidden"] + dim
    if kind == "predict":
        return {"bytes": n * (2.0 * d + 4.0 * dim) + 4.0 * params, "flops": 2.0 * n * per_row}
    if kind == "gradients":
        return {"bytes": n * 4.0 * (d + dim) + 8.0 * params, "flops": 6.0 * n * per_row}
    rows = case["steps"] * case["batch"]
    return {"bytes": rows * (2.0 * d + 4.0 * dim) + case["steps"] * 24.0 * params,
            "flops": 6.0 * rows * per_row}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _exact_graph(case, seed):
    """smooth_knn_dist, the membership weights and their fuzzy union in float64."""
    n, k = case["n"], case["k"]
    idx, dist, _ = _knn(n, case["d"], k, _gen(seed), False)
    idx = idx.cpu().numpy().astype(np.int64)
    d = dist.double()
    rho = d[:, :1]
    adj = (d - rho).clamp_min(0.0)
    target = math.log2(k)
    lo = torch.zeros_like(rho)
    hi = torch.full_like(rho, float("inf"))
    mid = torch.ones_like(rho)
    live = torch.ones_like(rho, dtype=torch.bool)
    for _ in range(64):
        val = torch.exp(-adj / mid).sum(1, keepdim=True)
        live = live & ((val - target).abs() >= 1e-5)
        up = val > target
        hi2 = torch.where(up, mid, hi)
        lo2 = torch.where(up, lo, mid)
        mid2 = torch.where(torch.isinf(hi2), 2.0 * mid, 0.5 * (lo2 + hi2))
        hi, lo = torch.where(live, hi2, hi), torch.where(live, lo2, lo)
        mid = torch.where(live, mid2, mid)
    w = torch.exp(-adj / mid).cpu().numpy()
    rows = np.repeat(np.arange(n, dtype=np.int64), k)
    cols, vals = idx.ravel(), w.ravel()
    if case["symmetrise"]:
        key = np.concatenate([rows * n + cols, cols * n + rows])
        val = np.concatenate([vals, vals])
        order = np.argsort(key, kind="stable")
        key, val = key[order], val[order]
        first = np.flatnonzero(np.concatenate([[True], key[1:] != key[:-1]]))
        a = val[first]
        two = np.diff(np.append(first, len(key))) == 2
        b = np.where(two, val[np.minimum(first + 1, len(val) - 1)], 0.0)
        vals = a + b - a * b
        keep = vals > 0.0
        key, vals = key[first][keep], vals[keep]
        rows, cols = key // n, key % n
    indptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=indptr[1:])
    cap = 2 * n * k
    return {"nnz": len(vals), "indptr": indptr,
            "indices": np.pad(cols, (0, cap - len(cols))).astype(np.uint32),
            "weights": np.pad(vals, (0, cap - len(vals)))}


def _exact_net(case, seed):
    w = torch.from_numpy(_weights(case, seed)).cuda().double()
    i, h, o = case["d"], case["hidden"], case["dim"]
    shapes = ((h, i), (h,), (h, h), (h,), (o, h), (o,))
    parts, at = [], 0
    for s in shapes:
        c = math.prod(s)
        parts.append(w[at:at + c].reshape(s))
        at += c
    return parts


def _exact_forward(p, x):
    a = torch.nn.functional.gelu(x @ p[0].T + p[1], approximate="tanh")
    a = torch.nn.functional.gelu(a @ p[2].T + p[3], approximate="tanh")
    return a @ p[4].T + p[5]


def exact(case, seed):
    kind = case["kind"]
    if kind == "graph":
        return _exact_graph(case, seed)
    if kind == "predict":
        p = _exact_net(case, seed)
        x, _ = _net_inputs(case, seed)
        return {"y": torch.cat([_exact_forward(p, c.double()) for c in x.split(65_536)])}
    if kind == "gradients":
        p = [q.clone().requires_grad_(True) for q in _exact_net(case, seed)]
        x, t = _net_inputs(case, seed)
        loss = (_exact_forward(p, x.double()) - t.double()).square().mean()
        loss.backward()
        return {"loss": float(loss.detach()),
                "grad": torch.cat([q.grad.reshape(-1) for q in p])}
    # The others have no such value. The embedding's epochs-per-sample schedule is defined by
    # its f32 recurrence (which edges fire, how many negatives they draw), and its trajectory,
    # like a training run's in BF16, parts from a 64-bit one after a few steps; the
    # label-propagation init thresholds and compares f32 vote sums and then embeds; the MST's
    # edges are whole numbers that follow from f32 distances.
    return None
