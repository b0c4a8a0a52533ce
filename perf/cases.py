"""The work that users of the partitioner have it do, as cases that can be timed.

Each case is one call of a public entry point of ``hunyuansc25_b200``:

* ``device``   ``Context.partition_device`` on a graph that is already on the GPU
* ``host``     ``Context.partition`` on host arrays (copies in and out included)
* ``batch``    ``Context.partition_prepared``: many independent graphs in one call
* ``nd``       ``Context.node_nd``: a nested-dissection ordering of a host graph
* ``edgecut``  ``Context.edgecut_device``: the cut of a partition a user holds
* ``mlp_grad`` ``Context.mlp_loss_grad``: one gradient of the move-scoring network

The graphs are those of the repository's workloads (2-D and 3-D grids, R-MAT with the
Graph500 quadrant probabilities, random geometric graphs of mean degree 12), drawn from
the seed on the GPU.  Partitions and orderings are deterministic integer results, so their
tolerance is "exact".
"""
import math
import os
import random

import numpy as np
import torch

import hunyuansc25_b200 as hp
from hunyuansc25_b200 import learn
from hunyuansc25_b200._abi import HP_MLP_NPARAM, default_options

TUNING_DIR = os.path.join(os.path.dirname(os.path.abspath(hp.__file__)), "tuning")


def listed():
    return [
        # the smallest of the workloads, resident on the GPU: launches and latency
        dict(name="grid2d_256_k8", call="device", graph="grid2d", x=256, y=256, k=8, ub=1.03, wmax=1),
        # a small power-law graph in a host program, the lower end of the batch workload's sizes
        dict(name="rmat_1500_k4_host", call="host", graph="rmat", n=1500, ef=8, k=4, ub=1.03, wmax=100),
        # the 3-D mesh workload (domain decomposition of a regular grid)
        dict(name="grid3d_128_k64", call="device", graph="grid3d", x=128, y=128, z=128, k=64, ub=1.03, wmax=10),
        # a ragged unit-weight mesh from a host program, odd number of parts with uneven targets
        dict(name="grid3d_97x61x83_k37_host", call="host", graph="grid3d", x=97, y=61, z=83, k=37, ub=1.05, wmax=1,
             plain_weights=True, uneven=True),
        # power-law graphs, plain refinement with the default tuning
        dict(name="rmat20_k256", call="device", graph="rmat", n=1 << 20, ef=16, k=256, ub=1.03, wmax=100),
        # the benchmark's workload: the largest power-law graph, learned move proposals, its own tuning file
        dict(name="rmat22_k256_learned", call="device", graph="rmat", n=1 << 22, ef=16, k=256, ub=1.03, wmax=100,
             learned=True, tuning="rmat22_learned"),
        # the largest geometric workload: many parts, low degrees, vertices in no particular order
        dict(name="rgg24_k1024", call="device", graph="rgg", n=1 << 24, k=1024, ub=1.05),
        # an ordinary geometric graph of odd size with vertex weights, from a host program
        dict(name="rgg_700001_k100_host", call="host", graph="rgg", n=700001, k=100, ub=1.03, vwmax=4),
        # a batch of uneven graphs (half grids, half R-MAT), the batch workload's sizes
        dict(name="batch_96", call="batch", count=96, nmin=1000, nmax=200000),
        # fill-reducing ordering of a 3-D mesh
        dict(name="nd_grid3d_40", call="nd", graph="grid3d", x=40, y=40, z=40, wmax=1),
        # evaluation of a partition a user holds
        dict(name="edgecut_rgg22_k256", call="edgecut", graph="rgg", n=1 << 22, k=256),
        # training of the move-scoring network: loss and gradient over a part of a move log
        dict(name="mlp_grad_300k", call="mlp_grad", n=300000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, nmax):
    kind = rng.choice(["grid2d", "grid3d", "rmat", "rgg"])
    n = _log_uniform(rng, 1000, nmax)
    if kind == "grid2d":
        x = max(2, int(round(math.sqrt(n) * math.exp(rng.uniform(-0.7, 0.7)))))
        return dict(graph=kind, x=x, y=max(2, n // x), wmax=rng.choice([1, 10, 100])), n
    if kind == "grid3d":
        x = max(2, int(round(n ** (1 / 3) * math.exp(rng.uniform(-0.5, 0.5)))))
        y = max(2, int(round(math.sqrt(n / x) * math.exp(rng.uniform(-0.5, 0.5)))))
        return dict(graph=kind, x=x, y=y, z=max(2, n // (x * y)), wmax=rng.choice([1, 10, 100])), n
    if kind == "rmat":
        n = min(n, 1 << 20)
        return dict(graph=kind, n=n, ef=rng.choice([8, 16]), wmax=rng.choice([1, 10, 100])), n
    return dict(graph=kind, n=n), n


def draw(rng: random.Random):
    call = rng.choice(["device", "device", "device", "host", "host", "batch", "nd", "edgecut", "mlp_grad"])
    if call == "batch":
        return dict(call=call, count=rng.randrange(8, 97), nmin=1000, nmax=rng.choice([20000, 50000, 200000]))
    if call == "mlp_grad":
        return dict(call=call, n=_log_uniform(rng, 4096, 1 << 20))
    if call == "nd":
        g, _ = _draw_graph(rng, 60000)
        while g["graph"] == "rmat":
            g, _ = _draw_graph(rng, 60000)
        return dict(g, call=call)
    g, n = _draw_graph(rng, 1 << 22)
    k = _log_uniform(rng, 2, max(2, min(1024, n // 64)))
    if call == "edgecut":
        return dict(g, call=call, k=k)
    c = dict(g, call=call, k=k, ub=rng.choice([1.03, 1.05, 1.1]))
    if rng.random() < 0.25:
        c["uneven"] = True
    if rng.random() < 0.25:
        c["vwmax"] = rng.choice([2, 4, 9])
    if g["graph"] == "rmat" and rng.random() < 0.4:
        c["learned"] = True
    return c


# ---- graphs, built on the GPU ----------------------------------------------------------

def _mix(x):
    """A 31-bit hash of non-negative int64 values (multiply and shift rounds)."""
    x = (x ^ (x >> 31)) * 0x2545F4914F6CDD1D
    x = (x ^ ((x >> 29) & 0x7FFFFFFFF)) * 0x369DEA0F31A53F85
    return (x >> 32) & 0x7FFFFFFF


def _edge_weights(u, v, seed, wmax):
    """Weights U{1..wmax}, the same in both directions of an edge."""
    if wmax <= 1:
        return torch.ones(u.numel(), dtype=torch.int32, device=u.device)
    key = torch.minimum(u, v) * 0x100000000 + torch.maximum(u, v) + (seed % 0x7FFFFFFF + 1) * 0x51ED270B
    return (_mix(key) % wmax + 1).to(torch.int32)


def _grid(dims, seed, wmax, dev):
    """Grid graph with 2 neighbours per dimension; dims from the slowest to the fastest."""
    n = math.prod(dims)
    v = torch.arange(n, dtype=torch.int64, device=dev)
    strides = [math.prod(dims[i + 1:]) for i in range(len(dims))]
    nbr, ok = [], []
    for s, d in zip(strides, dims):
        nbr.append(v - s)
        ok.append((v // s) % d > 0)
    for s, d in reversed(list(zip(strides, dims))):
        nbr.append(v + s)
        ok.append((v // s) % d < d - 1)
    nbr, ok = torch.stack(nbr, 1), torch.stack(ok, 1)
    xadj = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    xadj[1:] = torch.cumsum(ok.sum(1), 0)
    u, w = v[:, None].expand_as(nbr)[ok], nbr[ok]
    return xadj.to(torch.int32), w.to(torch.int32), _edge_weights(u, w, seed, wmax)


def _csr_from_keys(keys, n, seed, wmax, dev):
    """CSR of sorted unique keys u * n + v."""
    u, v = keys // n, keys % n
    xadj = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    xadj[1:] = torch.cumsum(torch.bincount(u, minlength=n), 0)
    return xadj.to(torch.int32), v.to(torch.int32), _edge_weights(u, v, seed, wmax)


def _rmat(n, ef, seed, wmax, dev, gen):
    scale = max(1, math.ceil(math.log2(n)))
    m = ef * n
    u = torch.zeros(m, dtype=torch.int64, device=dev)
    v = torch.zeros(m, dtype=torch.int64, device=dev)
    for _ in range(scale):
        r = torch.rand(m, device=dev, generator=gen)
        u = u * 2 + (r >= 0.76)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    keep = (u != v) & (u < n) & (v < n)
    u, v = u[keep], v[keep]
    keys = torch.unique(torch.cat([u * n + v, v * n + u]))
    return _csr_from_keys(keys, n, seed, wmax, dev)


def _rgg(n, dev, gen):
    """Random geometric graph of mean degree 12 in the unit square; w = int(1000 (1 - d/r)) + 1."""
    radius = math.sqrt(12.0 / (math.pi * n))
    p = torch.rand(2, n, device=dev, generator=gen, dtype=torch.float64)
    g = max(1, int(1.0 / radius))
    cx, cy = (p * g).long().clamp_(max=g - 1)
    order = torch.argsort(cy * g + cx)
    start = torch.zeros(g * g + 1, dtype=torch.int64, device=dev)
    start[1:] = torch.cumsum(torch.bincount(cy * g + cx, minlength=g * g), 0)
    keys, weights = [], []
    ids = torch.arange(n, device=dev)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            x, y = cx + dx, cy + dy
            inside = (x >= 0) & (x < g) & (y >= 0) & (y < g)
            i = ids[inside]
            cell = (y * g + x)[inside]
            count = start[cell + 1] - start[cell]
            first = torch.cumsum(count, 0) - count
            a = torch.repeat_interleave(i, count)
            at = torch.arange(a.numel(), device=dev) - torch.repeat_interleave(first - start[cell], count)
            b = order[at]
            d2 = (p[:, a] - p[:, b]).square().sum(0)
            near = (d2 < radius * radius) & (a != b)
            a, b, d2 = a[near], b[near], d2[near]
            keys.append(a * n + b)
            weights.append((1000.0 * (1.0 - d2.sqrt() / radius)).to(torch.int32) + 1)
    keys, at = torch.sort(torch.cat(keys))
    xadj, adj, _ = _csr_from_keys(keys, n, 0, 1, dev)
    return xadj, adj, torch.cat(weights)[at]


def _graph(case, seed, dev):
    """(xadj, adjncy, adjwgt) of the case, int32 CUDA tensors."""
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    kind = case["graph"]
    if kind == "grid2d":
        return _grid((case["y"], case["x"]), seed, case["wmax"], dev)
    if kind == "grid3d":
        return _grid((case["z"], case["y"], case["x"]), seed, case["wmax"], dev)
    if kind == "rmat":
        return _rmat(case["n"], case["ef"], seed, case["wmax"], dev, gen)
    return _rgg(case["n"], dev, gen)


def _size(case):
    """(vertices, adjacency entries): exact for grids, expected for the random graphs."""
    kind = case["graph"]
    if kind in ("grid2d", "grid3d"):
        dims = [case[d] for d in "xyz" if d in case]
        n = math.prod(dims)
        return n, sum(2 * (n // d) * (d - 1) for d in dims)
    if kind == "rmat":
        return case["n"], int(1.8 * case["ef"] * case["n"])   # about a tenth of the edges are repeats or loops
    return case["n"], 12 * case["n"]


def _targets(case):
    """Uneven target fractions: the last part is three times the first."""
    return np.linspace(1.0, 3.0, case["k"]).astype(np.float32) if case.get("uneven") else None


def _vertex_weights(case, seed, n, dev):
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed + 77)
    if case.get("vwmax", 1) > 1:
        return torch.randint(1, case["vwmax"] + 1, (n,), device=dev, generator=gen, dtype=torch.int32)
    grid = case["graph"] in ("grid2d", "grid3d")
    if grid and (case["wmax"] == 1 or case["call"] == "nd") and not case.get("plain_weights"):
        # another graph for each seed where the edges alone would always be the same
        return torch.randint(1, 3, (n,), device=dev, generator=gen, dtype=torch.int32)
    return torch.ones(n, dtype=torch.int32, device=dev)


def _host(g, vwgt):
    from hunyuansc25_b200.graphs import Graph
    xadj, adjncy, adjwgt = (t.cpu().numpy() for t in g)
    return Graph(xadj, adjncy, vwgt.cpu().numpy(), adjwgt)


def _batch_specs(case):
    """(kind, n, k) of the batch's graphs: the same sizes for every seed, log-uniform."""
    rng = random.Random(case["count"] * 7919 + case["nmax"])
    return [("grid2d" if i % 2 == 0 else "rmat", _log_uniform(rng, case["nmin"], case["nmax"]),
             rng.choice([2, 4, 8, 16, 32, 64])) for i in range(case["count"])]


def _batch_case(kind, n):
    if kind == "grid2d":
        x = max(1, int(round(math.sqrt(n))))
        return dict(graph="grid2d", x=x, y=max(1, int(round(n / x))), wmax=100)
    return dict(graph="rmat", n=n, ef=8, wmax=100)


def prepare(case, seed):
    dev = torch.device("cuda", 0)
    ctx = hp.Context(0)
    s = dict(case=case, ctx=ctx, opt=default_options())
    call = case["call"]
    if call == "batch":
        specs = _batch_specs(case)
        graphs = []
        for i, (kind, n, _) in enumerate(specs):
            g = _graph(_batch_case(kind, n), (seed * 1009 + i) % 0x7FFFFFFF, dev)
            graphs.append(_host(g, torch.ones(g[0].numel() - 1, dtype=torch.int32)))
        s["batch"] = ctx.prepare_batch(graphs, [k for _, _, k in specs], 1.03)
        return s
    if call == "mlp_grad":
        s["x"], s["y"] = _samples(case, seed, dev)
        ctx.mlp_set_params(learn.init_params(seed), 0.0)
        return s
    g = _graph(case, seed, dev)
    n = g[0].numel() - 1
    if call == "edgecut":
        gen = torch.Generator(device=dev)
        gen.manual_seed(seed + 5)
        s["g"] = g
        s["where"] = torch.randint(0, case["k"], (n,), device=dev, generator=gen, dtype=torch.int32)
        return s
    if case.get("learned"):
        s["opt"] = default_options(learned=1)
        params, threshold, _ = learn.load_params()
        ctx.mlp_set_params(params, threshold)
    if case.get("tuning"):
        ctx.load_tuning(os.path.join(TUNING_DIR, case["tuning"] + ".json"))
    vwgt = _vertex_weights(case, seed, n, dev)
    s["targets"] = _targets(case) if "k" in case else None
    if case.get("plain_weights"):
        # no weights are passed: another numbering of the same mesh for each seed
        g = _renumbered(g, seed, dev)
        s["host"] = _host(g, vwgt)
        s["host"].vwgt = s["host"].adjwgt = None
    elif call == "device":
        s["g"], s["vwgt"] = g, vwgt
        s["part"] = torch.empty(n, dtype=torch.int32, device=dev)
    else:
        s["host"] = _host(g, vwgt)
    return s


def _renumbered(g, seed, dev):
    """The graph with its vertices shifted cyclically by an amount drawn from the seed."""
    xadj, adjncy, adjwgt = g
    n = xadj.numel() - 1
    shift = random.Random(seed).randrange(n)
    deg = (xadj[1:] - xadj[:-1]).long()
    u = (torch.repeat_interleave(torch.arange(n, device=dev), deg) + shift) % n
    v = (adjncy.long() + shift) % n
    return _csr_from_keys(torch.sort(u * n + v).values, n, 0, 1, dev)


def _samples(case, seed, dev):
    """Features in the ranges that the refiner's candidates have, a fifth of them labelled 1."""
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    x = torch.rand(case["n"], 8, device=dev, generator=gen)
    x[:, 0] = x[:, 0] * 2 - 1
    x[:, 5:7] = x[:, 5:7] * 2 - 1
    x[:, 7] = (x[:, 7] < 0.4).float()
    y = (torch.rand(case["n"], device=dev, generator=gen) < 0.2).float()
    return x, y


def run(state):
    case, ctx = state["case"], state["ctx"]
    call = case["call"]
    if call == "device":
        xadj, adjncy, adjwgt = state["g"]
        return ctx.partition_device(xadj, adjncy, case["k"], state["vwgt"], adjwgt, case["ub"], state["targets"],
                                    state["opt"], part=state["part"])
    if call == "host":
        h = state["host"]
        return ctx.partition(h.xadj, h.adjncy, case["k"], h.vwgt, h.adjwgt, case["ub"], state["targets"],
                             state["opt"])
    if call == "batch":
        b = state["batch"]
        ctx.partition_prepared(b, state["opt"])
        return b.part, b.cuts
    if call == "nd":
        h = state["host"]
        return ctx.node_nd(h.xadj, h.adjncy, h.vwgt, state["opt"])
    if call == "edgecut":
        xadj, adjncy, adjwgt = state["g"]
        return ctx.edgecut_device(xadj, adjncy, adjwgt, state["where"])
    return ctx.mlp_loss_grad(state["x"], state["y"])


def work(case):
    """Bytes: the CSR, the weights and (edgecut) the partition read once, the results written once."""
    call = case["call"]
    if call == "mlp_grad":
        # forward 2, backward 4 operations per weight and sample
        return {"bytes": 36.0 * case["n"] + 8.0 * HP_MLP_NPARAM, "flops": 6.0 * HP_MLP_NPARAM * case["n"]}
    if call == "batch":
        total = 0
        for kind, n, _ in _batch_specs(case):
            nn, m = _size(_batch_case(kind, n))
            total += 12 * nn + 8 * m
        return {"bytes": float(total), "flops": 0.0}
    n, m = _size(case)
    if call == "edgecut":
        return {"bytes": 8.0 * n + 8.0 * m, "flops": float(m)}
    if call == "nd":
        return {"bytes": 16.0 * n + 4.0 * m, "flops": 0.0}
    weights = 0 if case.get("plain_weights") else 4 * n + 4 * m
    return {"bytes": 8.0 * n + 4.0 * m + weights, "flops": 0.0}


def tolerance(case):
    # integers throughout, and deterministic; the network's sums are 32-bit
    return {"rel": 1e-5, "max": 1e-4} if case["call"] == "mlp_grad" else "exact"


def exact(case, seed):
    """The cut by counting, the gradient in 64 bits; a partition or an ordering has no value of its own."""
    dev = torch.device("cuda", 0)
    if case["call"] == "edgecut":
        s = prepare(case, seed)
        xadj, adjncy, adjwgt = s["g"]
        where = s["where"]
        own = torch.repeat_interleave(where, (xadj[1:] - xadj[:-1]).long())
        return int(adjwgt.long()[own != where[adjncy.long()]].sum()) // 2
    if case["call"] != "mlp_grad":
        return None
    x, y = (t.double() for t in _samples(case, seed, dev))
    p = torch.from_numpy(learn.init_params(seed)).to(dev).double().requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = torch.split(p, [256, 32, 1024, 32, 32, 1])
    h = torch.relu(x @ w1.view(32, 8).T + b1)
    h = torch.relu(h @ w2.view(32, 32).T + b2)
    loss = torch.nn.functional.binary_cross_entropy_with_logits(h @ w3 + b3, y)
    loss.backward()
    return float(loss), p.grad.cpu().numpy()
