"""What a user of plant_gb300 has it do, as cases that can be timed.

Building exact labelings (the package's main path) of road-like, scale-free
and directed graphs; answering distance queries, from one pair to millions,
alone and through the server; computing the betweenness order; training and
running the learned ranking; reading a graph file.  Graph shapes are those of
the package's generators, tests and benchmark.
"""
from __future__ import annotations

import ctypes
import math
import tempfile

import numpy as np
import torch

import plant_gb300 as P

# Sizes: `side` is a grid's side (side * side vertices), `scale` the log2 of a
# power-law graph's vertices, `k` a number of query pairs.
ROAD_SIDES = (64, 512)
RMAT_SCALES = (11, 17)
DIRECTED_SCALES = (11, 15)


def listed():
    return [
        # labels of a small road-like grid under the degree order: latency of
        # a whole build (the 100 x 100 grid is the smallest benchmark graph)
        {"name": "build_road_100", "do": "build", "graph": "road", "side": 100, "order": "degree", "mode": "hybrid"},
        # labels of a road network of a quarter million vertices under the
        # sampled betweenness order, as a routing service builds them
        {"name": "build_road_512", "do": "build", "graph": "road", "side": 512, "order": "betweenness",
         "mode": "hybrid"},
        # labels of a scale-free (social, web) graph with unit lengths
        {"name": "build_rmat_17", "do": "build", "graph": "rmat", "scale": 17, "order": "degree", "mode": "hybrid"},
        # labels of a directed, weighted, skewed graph by the reference's own
        # schedule (run_paraPLL: pruned trees and a clean pass)
        {"name": "build_directed_15_gll", "do": "build", "graph": "directed", "scale": 15, "order": "degree",
         "mode": "gll"},
        # one distance, as an interactive caller asks it
        {"name": "query_1", "do": "query", "graph": "road", "side": 256, "k": 1},
        # one large request from host arrays
        {"name": "query_65536", "do": "query", "graph": "road", "side": 256, "k": 65536},
        # a bulk job on pairs and answers that stay on the device
        {"name": "query_device_4m", "do": "query_device", "graph": "road", "side": 256, "k": 4000037},
        # requests of mixed sizes in flight at once through the server
        {"name": "serve_48", "do": "serve", "graph": "rmat", "scale": 15, "requests": 48, "most": 16384},
        # the order a road-like graph is labelled under
        {"name": "order_road_256", "do": "order", "graph": "road", "side": 256, "sources": 256},
        # one training pass of the learned ranking on its largest training graph
        {"name": "rank_grad_15", "do": "rank_grad", "graph": "rmat", "scale": 15},
        # scores of the trained network for a large road-like graph
        {"name": "rank_predict_512", "do": "rank_predict", "graph": "road", "side": 512},
        # a DIMACS road file read into a graph
        {"name": "read_road_512", "do": "read", "graph": "road", "side": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["build", "build", "build", "query", "query_device", "serve", "order", "rank_grad",
                     "rank_predict", "read"])
    c = {"do": do}
    if do == "build":
        c["graph"] = rng.choice(["road", "rmat", "directed"])
    elif do in ("query", "query_device", "serve", "order", "rank_grad", "rank_predict"):
        c["graph"] = rng.choice(["road", "rmat"])
    else:
        c["graph"] = "road"
    whole = do in ("build", "rank_predict", "read")
    if c["graph"] == "road":
        c["side"] = _log(rng, ROAD_SIDES[0], ROAD_SIDES[1] if whole else 256)
    elif c["graph"] == "rmat":
        c["scale"] = rng.randint(RMAT_SCALES[0], RMAT_SCALES[1] if whole else 15)
        c["ef"] = rng.randint(6, 16)
    else:
        c["scale"] = rng.randint(*DIRECTED_SCALES)
        c["ef"] = rng.randint(4, 8)
    if do == "build":
        c["order"] = "betweenness" if c["graph"] == "road" and rng.random() < 0.6 else "degree"
        c["mode"] = rng.choice(["hybrid", "hybrid", "gll", "plant"])
        if c["order"] == "degree" and c["graph"] == "road":
            c["side"] = min(c["side"], 200)   # a degree order says little about a grid: its labels are several times larger
    elif do == "query":
        c["k"] = _log(rng, 1, 300000)
    elif do == "query_device":
        c["k"] = _log(rng, 100, 4000000)
    elif do == "serve":
        c["requests"] = rng.randint(1, 60)
        c["most"] = _log(rng, 16, 65536)
    elif do == "order":
        c["sources"] = rng.choice([32, 64, 256, 256])
    return c


# ------------------------------------------------------------------ inputs
def _edges(case, seed, highways=True):
    """Undirected edges (n, u, v, length) of the generators' shapes: a grid
    with 5% of its edges deleted, 1% diagonals and a few long highways, or a
    symmetrised RMAT graph.  Without highways a grid has the same number of
    edges for every seed."""
    rng = np.random.default_rng(seed)
    if case["graph"] == "road":
        side = case["side"]
        n = side * side
        i = np.arange(n, dtype=np.int64).reshape(side, side)
        uv = np.concatenate([np.stack([i[:, :-1].ravel(), i[:, 1:].ravel()], 1),
                             np.stack([i[:-1].ravel(), i[1:].ravel()], 1)])
        uv = uv[np.sort(rng.permutation(len(uv))[len(uv) // 20:])]
        diag = np.stack([i[:-1, :-1].ravel(), i[1:, 1:].ravel()], 1)
        uv = np.concatenate([uv, diag[rng.permutation(len(diag))[:n // 100]]])
        length = rng.integers(1, 1001, len(uv))
        if highways:
            k, reach = max(1, n // 524), max(2, min(64, side // 8))
            a = rng.integers(0, side, (k, 2))
            b = np.clip(a + rng.integers(-(reach // 2), reach // 2 + 1, (k, 2)), 0, side - 1)
            far = np.abs(a - b).sum(1)
            hw = np.stack([a[:, 0] * side + a[:, 1], b[:, 0] * side + b[:, 1]], 1)[far > 2]
            uv = np.concatenate([uv, hw])
            length = np.concatenate([length, 150 * far[far > 2]])
        return n, uv[:, 0], uv[:, 1], length.astype(np.int32)
    n = 1 << case["scale"]
    m = n * case.get("ef", 16)
    gen = torch.Generator().manual_seed(int(seed))
    uv = torch.zeros((m, 2), dtype=torch.int64)
    for _ in range(case["scale"]):
        r = torch.rand(m, generator=gen)
        uv[:, 0] = 2 * uv[:, 0] + (r >= 0.76)
        uv[:, 1] = 2 * uv[:, 1] + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    uv = np.sort(uv[uv[:, 0] != uv[:, 1]].numpy(), axis=1)
    uv = np.unique(uv[:, 0] * n + uv[:, 1])
    return n, uv // n, uv % n, np.ones(len(uv), np.int32)


def _graph(case, seed):
    if case["graph"] == "road":
        return P.Graph.from_arcs(*_edges(case, seed, case["do"] != "read"), undirected=True)
    if case["graph"] == "rmat":
        return P.Graph.rmat(case["scale"], case.get("ef", 16), seed=seed)
    # directed, weighted, skewed degrees: endpoints half uniform, half from a
    # Pareto tail over a permutation
    rng = np.random.default_rng(seed)
    n = 1 << case["scale"]
    m = n * case.get("ef", 8)
    perm = rng.permutation(n).astype(np.uint32)

    def ends():
        z = perm[np.minimum((rng.pareto(1.2, m) * 40).astype(np.int64), n - 1)]
        return np.where(rng.random(m) < 0.5, z, rng.integers(0, n, m).astype(np.uint32)).astype(np.uint32)

    src, dst = ends(), ends()
    keep = src != dst
    return P.Graph.from_arcs(n, src[keep], dst[keep], rng.integers(1, 100, m).astype(np.int32)[keep])


def _order(case, g, seed):
    if case.get("order", "betweenness" if case["graph"] == "road" else "degree") == "betweenness":
        return P.Order.betweenness(g, case.get("sources", 256), seed)
    return P.Order.degree(g, seed)


_MODES = {"hybrid": P.MODE_HYBRID, "gll": P.MODE_GLL, "plant": P.MODE_PLANT}


def _rank_input(case, seed):
    """Edges, a parameter vector and a target of the ranking network."""
    n, u, v, length = _edges(case, seed, False)
    rng = np.random.default_rng(seed + 1)

    def glorot(a, b, size):
        lim = math.sqrt(6.0 / (a + b))
        return rng.uniform(-lim, lim, size)

    parts = [glorot(3, 64, 3 * 64), rng.normal(0, 0.05, 64)]
    for _ in range(3):
        parts += [glorot(128, 64, 128 * 64), rng.normal(0, 0.05, 64)]
    parts += [glorot(64, 1, 64), np.zeros(1)]
    params = np.concatenate(parts).astype(np.float32)
    t = np.log1p(np.bincount(u, minlength=n) + np.bincount(v, minlength=n)) + 0.3 * rng.normal(size=n)
    target = ((t - t.mean()) / t.std()).astype(np.float32)
    return n, u, v, length, params, target


def prepare(case, seed):
    do = case["do"]
    s = {"case": case, "seed": seed}
    if do in ("rank_grad", "rank_predict"):
        n, u, v, length, params, target = _rank_input(case, seed)
        s["graph"] = P.Graph.from_arcs(n, u, v, length, undirected=True)
        s["net"] = P.RankNet(3)
        s["net"].set_params(params)
        s["target"] = target
        return s
    g = _graph(case, seed)
    if do == "read":
        s["file"] = tempfile.NamedTemporaryFile(suffix=".gr")   # removed with the state
        g.write(s["file"].name)
        return s
    s["graph"] = g
    if do == "order":
        return s
    s["order"] = _order(case, g, seed)
    g.to_device()
    if do == "build":
        # label arrays for the host, kept over builds (the number of labels
        # depends on the graph: room for the largest)
        n, room = _sizes(case)[0], int(2 * _sizes(case)[0] * _most_label(case))
        s["out"] = [np.zeros(2 * n + 1, np.int64), np.zeros(room, np.int32), np.zeros(room, np.int32)]
        for a in s["out"]:
            a.fill(0)
        return s
    s["labels"] = P.build(g, s["order"])
    n = g.get_n()
    if do == "query":
        s["pairs"] = P.generate_query(case["k"], n, seed=seed)
        P.query(s["labels"], s["pairs"][:1])
    elif do == "query_device":
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        s["pairs"] = torch.randint(0, n, (case["k"], 2), generator=gen, device="cuda", dtype=torch.int32)
        s["out"] = torch.empty(case["k"], dtype=torch.int32, device="cuda")
    else:
        rng = np.random.default_rng(seed)
        k = np.exp(np.random.default_rng(7).uniform(0, math.log(case["most"]), case["requests"])).astype(np.int64) + 1
        s["requests"] = [rng.integers(0, n, (int(x), 2)).astype(np.uint32) for x in k]
        s["server"] = P.Server(s["labels"])
    return s


def run(s):
    case = s["case"]
    do = case["do"]
    if do == "build":
        labels = P.build(s["graph"], s["order"], mode=_MODES[case["mode"]])
        off, hub, dist = s["out"]
        if labels.total() > len(hub):
            raise ValueError("%d labels: more than there is room for" % labels.total())
        rc = P.lib().chl_labels_export(labels._h, ctypes.cast(off.ctypes.data, ctypes.POINTER(ctypes.c_uint64)),
                                       ctypes.cast(hub.ctypes.data, ctypes.POINTER(ctypes.c_uint32)),
                                       ctypes.cast(dist.ctypes.data, ctypes.POINTER(ctypes.c_int32)))
        if rc != P.CHL_OK:
            raise P.CHLError(rc, "export")
        return s["out"]
    if do == "query":
        if case["k"] == 1:
            return s["labels"].query(int(s["pairs"][0, 0]), int(s["pairs"][0, 1]))
        return P.query(s["labels"], s["pairs"])
    if do == "query_device":
        rc = P.lib().chl_query_batch_device(s["labels"]._h, ctypes.c_void_p(s["pairs"].data_ptr()), case["k"],
                                            ctypes.c_void_p(s["out"].data_ptr()),
                                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != P.CHL_OK:
            raise P.CHLError(rc, "query")
        return s["out"]
    if do == "serve":
        srv = s["server"]
        ids = [srv.submit(q) for q in s["requests"]]
        return [srv.wait(i, len(q))[0] for i, q in zip(ids, s["requests"])]
    if do == "order":
        return P.Order.betweenness(s["graph"], case["sources"], s["seed"])
    if do == "rank_grad":
        loss, grads = s["net"].grad(s["graph"], s["target"])
        return {"loss": loss, "grads": grads}
    if do == "rank_predict":
        return s["net"].predict(s["graph"])
    g, _ = P.Graph.read_gpu(s["file"].name)
    off, head, length = g.csr()
    return [off.view(np.int64), head.view(np.int32), length]


# -------------------------------------------------------------------- work
def _sizes(case):
    """(vertices, arcs) of a case's graph, arcs counted in each direction."""
    if case["graph"] == "road":
        n = case["side"] ** 2
        return n, int(3.82 * n)
    if case["graph"] == "rmat":
        n = 1 << case["scale"]
        return n, int(2 * 0.88 * n * case.get("ef", 16))   # without duplicates
    n = 1 << case["scale"]
    return n, n * case.get("ef", 8)


def _avg_label(case):
    """Mean list length, about (measured over the declared sizes)."""
    if case["graph"] == "road":
        return 1.45 * case["side"] if case.get("order") == "degree" else 1.007 * case["side"] ** 0.934
    if case["graph"] == "rmat":
        return 22 * 1.292 ** (case["scale"] - 11) * (case.get("ef", 16) / 16) ** 0.5
    return 10.5


def _most_label(case):
    return 1.5 * _avg_label(case) + 10


def work(case):
    n, m = _sizes(case)
    do = case["do"]
    if do == "build":
        # the arcs once, and every label written: both lists of a vertex, 8 B an entry
        return {"bytes": 8 * m + 16 * n * _avg_label(case), "flops": 0}
    if do in ("query", "query_device"):
        return {"bytes": case["k"] * (16 * _avg_label(case) + 12), "flops": 0}
    if do == "serve":
        mean = case["most"] / max(1.0, math.log(case["most"]))   # of log-uniform sizes
        return {"bytes": case["requests"] * mean * (16 * _avg_label(case) + 12), "flops": 0}
    if do == "order":
        # per source: each arc read for distances, path counts and dependencies
        # (12 B each), and three values of each vertex written
        return {"bytes": min(case["sources"], n) * (36 * m + 20 * n), "flops": 0}
    if do == "read":
        return {"bytes": 17 * m + 16 * m + 16 * n, "flops": 0}
    # three layers: each vertex's 64 bf16 read and written, its neighbours' mean
    # written and read, the arcs once; a [n x 128] x [128 x 64] product each
    layers, flops = 3 * (n * 64 * 2 * 4 + 4 * m), 3 * 2 * n * 128 * 64
    if do == "rank_predict":
        return {"bytes": layers, "flops": flops}
    return {"bytes": 3 * layers, "flops": 3 * flops}


# ------------------------------------------------------------------- exact
def _mix(z):
    with np.errstate(over="ignore"):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _features(n, src, head, off, seed=1):
    """Standardised [log1p degree, log1p of the neighbours' degrees, sampled
    clustering] (a neighbour pair is closed if the second is among the first
    256 neighbours of the first)."""
    deg = np.diff(off)
    x = np.zeros((n, 3))
    x[:, 0] = np.log1p(2.0 * deg)
    x[:, 1] = np.log1p(np.bincount(src, weights=2.0 * deg[head], minlength=n))
    first = np.arange(len(head)) - off[src] < 256
    edges = src[first] * n + head[first]
    v = np.flatnonzero(deg >= 2)
    hit = np.zeros(len(v))
    d = deg[v].astype(np.uint64)
    for k in range(16):
        with np.errstate(over="ignore"):
            h = _mix(np.uint64(seed) ^ (v.astype(np.uint64) * np.uint64(0x100000001B3) + np.uint64(k)))
        i = (h % d).astype(np.int64)
        j = ((h >> np.uint64(32)) % (d - np.uint64(1))).astype(np.int64)
        j += j >= i
        e = head[off[v] + i] * n + head[off[v] + j]
        at = np.minimum(np.searchsorted(edges, e), len(edges) - 1)
        hit += edges[at] == e
    x[v, 2] = hit / 16
    x = x.astype(np.float32).astype(np.float64)
    sd = x.std(axis=0)
    return (x - x.mean(axis=0)) * np.where(sd > 1e-12, 1 / np.maximum(sd, 1e-12), 0.0)


def exact(case, seed):
    if case["do"] not in ("rank_grad", "rank_predict"):
        return None   # whole numbers
    n, u, v, _, params, target = _rank_input(case, seed)
    key = np.sort(np.concatenate([u * n + v, v * n + u]))
    src, head = key // n, key % n
    off = np.searchsorted(src, np.arange(n + 1))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.from_numpy(_features(n, src, head, off)).to(dev)
    inv = torch.from_numpy(1.0 / np.maximum(np.diff(off), 1)).to(dev)[:, None]
    S, T = torch.from_numpy(src).to(dev), torch.from_numpy(head).to(dev)
    p = torch.from_numpy(params.astype(np.float64)).to(dev)
    grad = case["do"] == "rank_grad"
    p.requires_grad_(grad)
    at = 0

    def take(*shape):
        nonlocal at
        k = math.prod(shape)
        at += k
        return p[at - k:at].reshape(shape)

    with torch.set_grad_enabled(grad):
        W, b = take(3, 64), take(64)
        h = torch.relu(x @ W + b)
        for _ in range(3):
            W, b = take(128, 64), take(64)
            m = torch.zeros_like(h).index_add(0, S, h[T]) * inv
            h = torch.relu(torch.cat([h, m], 1) @ W + b)
        w, c = take(64), take(1)
        score = h @ w + c
        if not grad:
            return score.cpu().numpy()
        loss = (score - torch.from_numpy(target.astype(np.float64)).to(dev)).square().mean()
        loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad.cpu().numpy()}
