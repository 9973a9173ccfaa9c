"""The work that users of this framework have it do, as cases that can be timed.

Every case goes through the public entry points of ``gstore_b200``: edge lists
are converted once (``Context.convert``), a query state is made once
(``Graph.state``) and a pass is what a program repeats on them, results
included: reset to the next query, run, take the result into a pinned host
array.  Graphs are R-MAT graphs with the Graph500 quadrant probabilities
(0.57, 0.19, 0.19, 0.05) and scrambled vertex ids, or uniform random ones,
made here with torch so that the 64-bit values of ``exact`` need nothing of
the framework.

* ``listed()``  the cases by name
* ``draw(rng)`` one more case of the same ranges
* ``prepare``, ``run``, ``work``, ``exact``  as their docstrings say
"""
import ctypes
import math
import random

import numpy as np
import torch

import gstore_b200 as gs


def _graph(vertices, edgefactor, directed=False, kind="rmat"):
    return {"vertices": vertices, "edgefactor": edgefactor, "directed": directed, "graph": kind}


def listed():
    """The cases by name; the comments say what each stands for in use."""
    return [
        # a query on a small graph: a few short sweeps, launches and host round trips count
        {"name": "bfs_small", "algo": "bfs", **_graph(1 << 16, 16)},
        # a crawl-like directed graph, vertex count no multiple of a tile window
        {"name": "bfs_directed", "algo": "bfs", **_graph(1_500_007, 8, True)},
        # the headline: BFS over Graph500 scale 26, edge factor 16, records far beyond L2
        {"name": "bfs_kron26", "algo": "bfs", **_graph(1 << 26, 16)},
        # the PageRank workload: 5 iterations on scale 20, edge factor 16
        {"name": "pagerank_kron20", "algo": "pagerank", "arg": 5, **_graph(1 << 20, 16)},
        # the same on a graph whose rank vectors alone fill half of L2
        {"name": "pagerank_kron24", "algo": "pagerank", "arg": 5, **_graph(1 << 24, 16)},
        # a directed graph without hubs: ten iterations, odd sizes, no locality to lean on
        {"name": "pagerank_uniform", "algo": "pagerank", "arg": 10, **_graph(3_000_017, 8, True, "uniform")},
        # components and cores of a large graph
        {"name": "wcc_kron25", "algo": "wcc", **_graph(1 << 25, 16)},
        {"name": "kcore_kron25", "algo": "kcore", "arg": 8, **_graph(1 << 25, 16)},
        # a new edge list on the device: converted to tiles, queried once, dropped
        {"name": "ingest_kron22", "algo": "ingest", **_graph(1 << 22, 16)},
        # 64 roots on one graph, with components and cores of it beside them, as one batch
        {"name": "batch_kron22", "algo": "batch", "roots": 64, "cores": 4, **_graph(1 << 22, 16)},
        # a burst of mixed requests to a server over three graphs (sizes given: the largest)
        {"name": "serve_burst", "algo": "serve", "requests": 32, **_graph(1 << 20, 16)},
        # the semi-external mode: records in pinned host memory, two segments in HBM
        {"name": "stream_kron22", "algo": "stream", "segment_mb": 32, **_graph(1 << 22, 16)},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any of the paths, sizes over the logarithm of their
    ranges, most of them no power of two."""
    algo = rng.choice(["bfs", "bfs", "pagerank", "pagerank", "wcc", "kcore", "ingest", "batch", "serve", "stream"])
    ef = rng.choice([2, 4, 8, 16, 16, 32])
    # the largest edge count of each path, so that no drawn case costs more
    # than the largest listed one
    most = {"bfs": 1 << 28, "pagerank": 1 << 27, "wcc": 1 << 28, "kcore": 1 << 28, "ingest": 1 << 25,
            "batch": 1 << 25, "serve": 1 << 23, "stream": 1 << 25}[algo]
    vertices = _log_uniform(rng, 20_000, most // ef)
    if rng.random() < 0.25:
        vertices = 1 << (vertices.bit_length() - 1)
    case = {"algo": algo,
            **_graph(vertices, ef, algo not in ("kcore", "batch", "serve") and rng.random() < 0.3,
                     "uniform" if rng.random() < 0.2 else "rmat")}
    if algo == "pagerank":
        case["arg"] = rng.choice([1, 3, 5, 10, 20])
    elif algo == "kcore":
        case["arg"] = rng.randint(2, 24)
    elif algo == "batch":
        case["roots"] = rng.randint(2, 64)
        case["cores"] = rng.randint(0, 4)
    elif algo == "serve":
        case["requests"] = rng.randint(8, 32)
    elif algo == "stream":
        case["segment_mb"] = rng.choice([4, 16, 32])
    return case


# ---------------------------------------------------------------- inputs --
def _edges(vertices, edgefactor, kind, seed):
    """(m, 2) int32 endpoint pairs on the GPU."""
    m = vertices * edgefactor
    gen = torch.Generator(device="cuda").manual_seed(seed)
    out = torch.empty((m, 2), dtype=torch.int32, device="cuda")
    if kind == "uniform":
        return out.random_(0, vertices, generator=gen)
    scale = max(1, (vertices - 1).bit_length())
    mask = (1 << scale) - 1
    keys = random.Random(seed)
    odd = [keys.randrange(mask + 1) | 1 for _ in range(2)]
    half = scale // 2 + 1

    def scramble(v):   # one to one on [0, 2^scale), then folded below `vertices`
        v.mul_(odd[0]).bitwise_and_(mask)
        v.bitwise_xor_(v >> half)
        v.mul_(odd[1]).bitwise_and_(mask)
        v.bitwise_xor_(v >> half)
        return v.remainder_(vertices)

    for lo in range(0, m, 1 << 25):
        n = min(1 << 25, m - lo)
        src = torch.zeros(n, dtype=torch.int32, device="cuda")
        dst = torch.zeros(n, dtype=torch.int32, device="cuda")
        u = torch.empty(n, device="cuda")
        for _ in range(scale):
            u.uniform_(generator=gen)
            down = u >= 0.76                                  # the quadrant's row
            right = ((u >= 0.57) & ~down) | (u >= 0.95)       # and its column
            src.mul_(2).add_(down)
            dst.mul_(2).add_(right)
        out[lo:lo + n, 0] = scramble(src)
        out[lo:lo + n, 1] = scramble(dst)
    return out


def _sizes(case):
    """Vertex counts and edge factors of the case's graphs (a server's three
    graphs go down by a factor of two and four)."""
    v, ef = case["vertices"], case["edgefactor"]
    if case["algo"] != "serve":
        return [(v, ef)]
    return [(v, ef), (max(1000, v // 2), ef), (max(1000, v // 4), 2 * ef)]


def _roots(pairs, n, seed):
    """n vertices that have an edge to another vertex."""
    at = torch.tensor([random.Random(seed).randrange(pairs.shape[0]) for _ in range(4 * n + 64)], device="cuda")
    some = pairs[at].cpu()
    return [int(a) for a, b in some.tolist() if a != b][:n]


def _requests(case, seed, roots):
    """(graph, algorithm, argument) of a server's burst."""
    rng = random.Random(seed)
    left = [list(r) for r in roots]
    out = []
    for i in range(case["requests"]):
        g = i % len(left)
        kind = i % 16
        if kind == 5:
            out.append((g, "wcc", 0))
        elif kind == 9:
            out.append((g, "kcore", rng.randint(4, 16)))
        elif kind == 14:
            out.append((g, "pagerank", 5))
        else:
            out.append((g, "bfs", left[g].pop()))
    return out


def _pinned(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()


def prepare(case, seed):
    """A program before its query: context, resident graph and query state (or
    batch inputs, server, host records), and the host array for the result."""
    algo = case["algo"]
    ctx = gs.Context(directed=case["directed"])
    state = {"algo": algo, "ctx": ctx}
    graphs, roots = [], []
    for k, (v, ef) in enumerate(_sizes(case)):
        pairs = _edges(v, ef, case["graph"], seed + 1000 * k)
        roots.append(_roots(pairs, max(case.get("roots", 1), case.get("requests", 1)), seed + k))
        torch.cuda.synchronize()
        if algo == "ingest":
            state["pairs"] = pairs
            break
        graphs.append(ctx.convert(pairs.data_ptr(), v, n_pairs=pairs.shape[0]))
    state["V"] = V = case["vertices"]
    if algo == "ingest":
        state["root"] = roots[0][0]
        state["out"] = _pinned(V, torch.uint8)
        return state
    del pairs
    torch.cuda.empty_cache()
    if algo == "serve":
        state["server"] = gs.Server(ctx)
        state["ids"] = [state["server"].add_graph(g) for g in graphs]
        state["requests"] = _requests(case, seed, roots)
        state["server"].reserve_host(8 * V * len(state["requests"]))
        return state
    graph = graphs[0]
    if algo == "batch":
        state["graph"], state["roots"] = graph, roots[0]
        state["ks"] = [4 + 4 * i for i in range(case["cores"])]
        state["depth"] = _pinned((len(roots[0]), V), torch.uint8)
        state["labels"] = _pinned(V, torch.int32)
        state["cores"] = _pinned((max(1, len(state["ks"])), V), torch.int32)
        return state
    if algo == "stream":
        start, grid, degree = graph.download()
        records = _pinned(grid.size, torch.int32).view(np.uint32)
        records[:] = grid
        graph.free()
        graph = ctx.upload_streamed(start, records, degree, V, case["segment_mb"] << 20)
        algo = "bfs"
    state["graph"] = graph
    state["arg"] = roots[0][0] if algo == "bfs" else case.get("arg", 0)
    state["query"] = graph.state(algo, state["arg"])
    dtype = {"bfs": torch.uint8, "pagerank": torch.float32, "wcc": torch.int32, "kcore": torch.int32}[algo]
    state["out"] = _pinned(V, dtype)
    return state


# ------------------------------------------------------------------ pass --
def _run_batch(state):
    ctx, graph, V = state["ctx"], state["graph"], state["V"]
    take = gs.lib().gs_batch_download

    def into(batch, query, row):
        ctx._check(take(batch._h, query, 0, row.ctypes.data_as(ctypes.c_void_p), row.nbytes))

    with gs.Batch(ctx) as batch:
        bfs = [batch.add(graph, "bfs", r) for r in state["roots"]]
        wcc = batch.add(graph, "wcc")
        cores = [batch.add(graph, "kcore", k) for k in state["ks"]]
        batch.run()
        for q, row in zip(bfs, state["depth"]):
            into(batch, q, row)
        into(batch, wcc, state["labels"])
        for q, row in zip(cores, state["cores"]):
            into(batch, q, row)
    return [state["depth"], state["labels"], state["cores"][:len(cores)] if cores else None]


def _run_server(state):
    server, ids = state["server"], state["ids"]
    rids = [server.submit(ids[g], algo, arg) for g, algo, arg in state["requests"]]
    left = len(rids)
    while left:
        server.step()
        left -= len(server.completed())
    return [server.result(r)[0] for r in rids]


def run(state):
    """One pass: the query and its whole result on the host."""
    algo = state["algo"]
    if algo == "batch":
        return _run_batch(state)
    if algo == "serve":
        return _run_server(state)
    if algo == "ingest":
        pairs = state["pairs"]
        graph = state["ctx"].convert(pairs.data_ptr(), state["V"], n_pairs=pairs.shape[0])
        with graph.state("bfs", state["root"]) as query:
            query.run()
            query.download_into(state["out"])
        degree = graph.degree()
        graph.free()
        return [state["out"], degree]
    query = state["query"]
    query.reset(state["arg"])
    query.run()
    return query.download_into(state["out"])


def work(case):
    """Bytes and operations of one pass that it cannot do without: the records
    (4 bytes each; an edge list has 8) once per query or iteration, the result."""
    out = {"bytes": 0.0, "flops": 0.0}
    algo = case["algo"]
    for v, ef in _sizes(case):
        e = v * ef
        if algo in ("bfs", "stream"):
            n = 4 * e + v
        elif algo == "pagerank":
            n = case["arg"] * (4 * e + 8 * v) + 4 * v
            out["flops"] += case["arg"] * (1 if case["directed"] else 2) * e
        elif algo in ("wcc", "kcore"):
            n = 4 * e + 4 * v
        elif algo == "ingest":
            n = 8 * e + 4 * e + 5 * v
        elif algo == "batch":
            n = (2 + case["cores"]) * 4 * e + (case["roots"] + 4 + 4 * case["cores"]) * v
        else:
            n = 4 * (4 * e) + case["requests"] // 3 * v
        out["bytes"] += n
    return out


# ----------------------------------------------------------------- exact --
def _pagerank64(pairs, vertices, iterations, directed):
    """rank = 0.15 + 0.85 sum of x over the in-edges, x = rank / degree, from
    x = 1 / V; self-loops are no edges, repeated edges count each time."""
    src, dst = pairs[:, 0], pairs[:, 1]
    keep = src != dst
    src, dst = src[keep], dst[keep]
    ones = torch.ones(1, dtype=torch.float64, device="cuda")

    def push(values, into, frm, to):
        for lo in range(0, frm.numel(), 1 << 25):
            t = to[lo:lo + (1 << 25)].long()
            into.index_add_(0, t, ones.expand(t.numel()) if values is None else values[frm[lo:lo + (1 << 25)].long()])

    degree = torch.zeros(vertices, dtype=torch.float64, device="cuda")
    push(None, degree, src, src)
    if not directed:
        push(None, degree, dst, dst)
    x = torch.full((vertices,), 1.0 / vertices, dtype=torch.float64, device="cuda")
    for _ in range(iterations):
        s = torch.zeros(vertices, dtype=torch.float64, device="cuda")
        push(x, s, src, dst)
        if not directed:
            push(x, s, dst, src)
        rank = 0.15 + 0.85 * s
        x = torch.where(degree > 0, rank / degree.clamp(min=1), torch.zeros_like(rank))
    return rank.cpu().numpy()


def exact(case, seed):
    """PageRank in 64 bits; every other result is a whole number."""
    if case["algo"] == "pagerank":
        pairs = _edges(case["vertices"], case["edgefactor"], case["graph"], seed)
        return _pagerank64(pairs, case["vertices"], case["arg"], case["directed"])
    if case["algo"] != "serve":
        return None
    edges = [_edges(v, ef, case["graph"], seed + 1000 * k) for k, (v, ef) in enumerate(_sizes(case))]
    roots = [_roots(p, max(case.get("roots", 1), case["requests"]), seed + k) for k, p in enumerate(edges)]
    return [_pagerank64(edges[g], edges_v, arg, False) if algo == "pagerank" else None
            for g, algo, arg in _requests(case, seed, roots)
            for edges_v in [_sizes(case)[g][0]]]
