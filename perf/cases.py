"""The workloads whose speed this repository is measured by.

Each case is work that a user of the engine has it do through the Python API:
a traversal (BFS, SSSP, CC) or a PageRank on a graph that is resident on the
GPU, many sources or seeds at once through the batched engine, and a whole
application from host arrays to host results.  ``listed()`` holds the fixed
cases, ``draw()`` gives more of the same ranges, ``prepare()`` makes a case's
inputs from a seed, ``run()`` is one pass, ``work()`` the least data it moves
and ``exact()`` its floating results in 64 bits without the engine.

Graphs are seeded synthetic ones made on the GPU: R-MAT with the quadrant
probabilities (0.57, 0.19, 0.19, 0.05), or uniform Erdos-Renyi; self loops
and duplicate edges are removed, the edge list is sorted by (src, dst).
"""
import random

import numpy as np
import torch

from graphreduce_gb300 import Batch, GASEngineGPU
from graphreduce_gb300.engine import initial_vertex_data
from graphreduce_gb300.learn import DATA, MLP

DEVICE = "cuda"
DAMPING, TOL = 0.85, 1e-6
ISLAND_SIDE = 32  # grid islands of the connected-component graphs: 32 x 32 vertices
MAX_SAMPLES = 1 << 26  # edge samples of the largest drawn graph


def listed():
    return [
        # BFS from one source on a small social-type graph: a latency-bound query
        {"name": "bfs_rmat16", "kind": "bfs", "graph": "rmat", "vertices": 1 << 16,
         "edge_factor": 16, "symmetric": True, "schedule": "auto"},
        # BFS from one source at the size of a large crawl
        {"name": "bfs_rmat22", "kind": "bfs", "graph": "rmat", "vertices": 1 << 22,
         "edge_factor": 16, "symmetric": True, "schedule": "auto"},
        # shortest paths on a tiny graph: launches and loop control are all there is
        {"name": "sssp_rmat12", "kind": "sssp", "graph": "rmat", "vertices": 4093,
         "edge_factor": 8, "symmetric": True, "schedule": "auto"},
        # shortest paths on a uniform graph of odd size: many similar rows, no hubs,
        # the fixed heuristic's push and pull iterations
        {"name": "sssp_er_odd", "kind": "sssp", "graph": "er", "vertices": 1499977,
         "edge_factor": 12, "symmetric": False, "schedule": "auto"},
        # shortest paths from one source at scale, the trained schedule
        {"name": "sssp_rmat22", "kind": "sssp", "graph": "rmat", "vertices": 1 << 22,
         "edge_factor": 16, "symmetric": True, "schedule": "learned"},
        # connected components at scale with 4,096 grid islands: a few heavy
        # iterations, then a long tail of light ones
        {"name": "cc_rmat22_islands", "kind": "cc", "graph": "rmat", "vertices": 1 << 22,
         "edge_factor": 16, "symmetric": True, "schedule": "learned", "islands": 4096},
        # precision PageRank of a directed web-type graph of 260 M edges
        {"name": "pagerank_rmat24", "kind": "pagerank", "graph": "rmat", "vertices": 1 << 24,
         "edge_factor": 16, "symmetric": False},
        # the reference application's PageRank (active sets, the general gather /
        # apply / scatter iteration that user programs take too)
        {"name": "pagerank_app_rmat18", "kind": "pagerank_app", "graph": "rmat",
         "vertices": 200003, "edge_factor": 16, "symmetric": False},
        # eight sources of shortest paths as the lanes of one batched run
        {"name": "lanes_sssp8_rmat22", "kind": "lanes", "what": "sssp", "lanes": 8, "graphs": 1,
         "min_vertices": 1 << 22, "max_vertices": 1 << 22, "edge_factor": 16},
        # many graphs of uneven size, 16 BFS sources each
        {"name": "batch_bfs16", "kind": "lanes", "what": "bfs", "lanes": 16, "graphs": 16,
         "min_vertices": 4097, "max_vertices": 600011, "edge_factor": 16},
        # the same graphs, 16 personalized-PageRank seeds each
        {"name": "batch_ppr16", "kind": "lanes", "what": "ppr", "lanes": 16, "graphs": 16,
         "min_vertices": 4097, "max_vertices": 600011, "edge_factor": 16},
        # a whole application: host edge list in, graph built, run(), host results out
        {"name": "app_sssp_rmat20", "kind": "app", "program": "sssp", "graph": "rmat",
         "vertices": 1 << 20, "edge_factor": 16, "symmetric": True},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng: random.Random):
    kind = rng.choice(["bfs", "bfs", "sssp", "sssp", "cc", "cc", "pagerank", "pagerank_app",
                       "lanes", "lanes", "lanes", "app"])
    ef = rng.randint(4, 32)
    graph = rng.choice(["rmat", "rmat", "er"])
    if kind == "lanes":
        what = rng.choice(["sssp", "bfs", "ppr"])
        lanes = rng.randint(1, 32)
        graphs = rng.choice([1, 1, 3, 8, 17])
        top = min(1 << 22, (1 << 22) * 8 * 16 // (max(8, lanes) * max(8, ef)))
        if what == "ppr":
            top = min(top, 1 << 19)
        big = _log_uniform(rng, 2000, max(4000, top // graphs))
        small = _log_uniform(rng, 1000, big) if graphs > 1 else big
        return {"kind": kind, "what": what, "lanes": lanes, "graphs": graphs,
                "min_vertices": min(small, big), "max_vertices": big, "edge_factor": ef}
    top = MAX_SAMPLES // ef
    if kind == "pagerank_app":
        top = min(top, 1 << 19)
    elif kind == "app":
        top = min(top, (1 << 24) // ef)
    vertices = _log_uniform(rng, 1000, min(top, 1 << 22))
    case = {"kind": kind, "graph": graph, "vertices": vertices, "edge_factor": ef,
            "symmetric": kind not in ("pagerank", "pagerank_app") and rng.random() < 0.75}
    if kind in ("bfs", "sssp", "cc"):
        case["schedule"] = rng.choice(["auto", "learned"])
    if kind == "cc" and rng.random() < 0.5:
        case["islands"] = _log_uniform(rng, 1, max(2, vertices // 1024))
    if kind == "app":
        case["program"] = rng.choice(["bfs", "sssp", "cc"])
    return case


# ---------------------------------------------------------------------------
# graphs
# ---------------------------------------------------------------------------
def _edges(graph, vertices, samples, seed, symmetric):
    """(src, dst) int32 on the GPU, sorted by (src, dst), no loops or duplicates."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    if graph == "er":
        s = torch.randint(vertices, (samples,), generator=gen, device=DEVICE)
        d = torch.randint(vertices, (samples,), generator=gen, device=DEVICE)
    else:
        s = torch.zeros(samples, dtype=torch.int64, device=DEVICE)
        d = torch.zeros(samples, dtype=torch.int64, device=DEVICE)
        for _ in range(max(1, (vertices - 1).bit_length())):
            u = torch.rand(samples, generator=gen, device=DEVICE)
            low = u >= 0.76  # quadrants c (0.76..0.95) and d (0.95..1)
            s.mul_(2).add_(low)
            d.mul_(2).add_(((u >= 0.57) & ~low) | (u >= 0.95))
        if vertices & (vertices - 1):
            s.remainder_(vertices)
            d.remainder_(vertices)
    keep = s != d
    s, d = s[keep], d[keep]
    key = s * vertices + d
    if symmetric:
        key = torch.cat([key, d * vertices + s])
    del s, d, keep
    key = torch.unique(key)
    src = torch.div(key, vertices, rounding_mode="floor")
    dst = key - src * vertices
    return src.to(torch.int32), dst.to(torch.int32)


def _with_islands(src, dst, vertices, islands):
    """Disjoint 32 x 32 four-neighbour grids (both directions) after the vertices."""
    k = ISLAND_SIDE
    at = torch.arange(k * k, device=DEVICE).view(k, k)
    a = torch.cat([at[:, :-1].reshape(-1), at[:-1, :].reshape(-1)])
    b = torch.cat([at[:, 1:].reshape(-1), at[1:, :].reshape(-1)])
    a, b = torch.cat([a, b]), torch.cat([b, a])
    first = vertices + k * k * torch.arange(islands, device=DEVICE).view(-1, 1)
    src = torch.cat([src, (first + a).reshape(-1).to(torch.int32)])
    dst = torch.cat([dst, (first + b).reshape(-1).to(torch.int32)])
    return src, dst, vertices + islands * k * k


def _weights(src, dst, seed):
    """Uniform in [1, 64], the same for both directions of an edge."""
    lo, hi = torch.minimum(src, dst).long(), torch.maximum(src, dst).long()
    h = (lo * 0x9E3779B1 + hi * 0x85EBCA77 + (seed & 0xFFFF) * 0xC2B2AE3D) & 0x7FFFFFFF
    h = ((h ^ (h >> 15)) * 0x2C1B3C6D) & 0x7FFFFFFF
    h = ((h ^ (h >> 12)) * 0x297A2D39) & 0x7FFFFFFF
    return (1 + ((h >> 8) & 63)).to(torch.int32)


def _pick(src, count, seed):
    """Vertices with out-edges: the sources of edges drawn uniformly."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed + 77)
    return src[torch.randint(src.shape[0], (count,), generator=gen, device=DEVICE)].cpu().numpy()


def _case_edges(case, seed):
    src, dst = _edges(case["graph"], case["vertices"], case["vertices"] * case["edge_factor"],
                      seed, case["symmetric"])
    vertices = case["vertices"]
    if case.get("islands"):
        src, dst, vertices = _with_islands(src, dst, vertices, case["islands"])
    return src, dst, vertices


def _lane_sizes(case):
    """Vertices of each graph, spread evenly over the logarithm of the range."""
    n, lo, hi = case["graphs"], case["min_vertices"], case["max_vertices"]
    if n == 1:
        return [hi]
    return [int(round(lo * (hi / lo) ** (i / (n - 1)))) for i in range(n)]


def _lane_graphs(case, seed):
    """[(vertices, src, dst)] and the sources or seeds [graphs][lanes]."""
    graphs, ids = [], []
    for i, v in enumerate(_lane_sizes(case)):
        src, dst = _edges("rmat", v, v * case["edge_factor"], seed * 64 + i, True)
        graphs.append((v, src, dst))
        ids.append(_pick(src, case["lanes"], seed * 64 + i))
    return graphs, np.stack(ids).astype(np.int32)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "lanes":
        graphs, ids = _lane_graphs(case, seed)
        batch = Batch()
        for v, src, dst in graphs:
            w = _weights(src, dst, seed).cpu().numpy() if case["what"] == "sssp" else None
            batch.add_graph(v, src.cpu().numpy(), dst.cpu().numpy(), w)
        batch.build()
        dtype = torch.float32 if case["what"] == "ppr" else torch.int32
        out = torch.empty((batch.num_vertices, case["lanes"]), dtype=dtype, device=DEVICE)
        return {"kind": kind, "what": case["what"], "batch": batch, "ids": ids, "out": out}

    src, dst, n = _case_edges(case, seed)
    program = {"pagerank_app": "pagerank", "app": case.get("program")}.get(kind, kind)
    source = int(_pick(src, 1, seed)[0])
    hsrc, hdst = src.cpu().numpy(), dst.cpu().numpy()
    w = _weights(src, dst, seed).cpu().numpy() if program == "sssp" else None
    outdeg = np.bincount(hsrc, minlength=n).astype(np.int32) if program == "pagerank" else None
    init = initial_vertex_data(program, n, source, outdeg)
    active = (source, source + 1) if program == "bfs" else (0, n)
    if kind == "app":
        return {"kind": kind, "program": program, "n": n, "src": hsrc, "dst": hdst, "w": w,
                "init": init, "active": active}

    engine = GASEngineGPU(program)
    engine.setGraph(n, init, len(hsrc), w, hsrc, hdst)
    state = {"kind": kind, "engine": engine, "active": active}
    if kind == "pagerank":
        state["out"] = torch.empty(n, dtype=torch.float32, device=DEVICE)
        return state
    raw = torch.from_numpy(init.view(np.int32).reshape(n, -1).copy())
    state["init"] = raw.to(DEVICE)
    state["out"] = torch.empty_like(state["init"])
    state["schedule"] = case.get("schedule", "auto")
    if state["schedule"] == "learned":
        engine.set_schedule_model(MLP.load(DATA / "schedule_head.npz"))
    return state


def run(state):
    kind = state["kind"]
    if kind == "lanes":
        out, ids = state["out"], state["ids"]
        if state["what"] == "ppr":
            state["batch"].run(ppr_seeds=ids, damping=DAMPING, tol=TOL, rank_out=out.data_ptr())
            return {"rank": out}
        if state["what"] == "bfs":
            r = state["batch"].run(bfs_sources=ids, depth_out=out.data_ptr())
            return {"depth": out, "levels": r.stats.bfs_iterations}
        r = state["batch"].run(sssp_sources=ids, dist_out=out.data_ptr())
        return {"dist": out, "iterations": r.stats.sssp_iterations}
    if kind == "app":
        data = state["init"].copy()
        engine = GASEngineGPU(state["program"])
        engine.setGraph(state["n"], data, len(state["src"]), state["w"], state["src"],
                        state["dst"])
        engine.setActive(*state["active"])
        iterations = engine.run()
        engine.getResults()
        engine.close()
        return {"vertex_data": data, "iterations": iterations}

    engine, out = state["engine"], state["out"]
    if kind == "pagerank":
        engine.pagerank_precision(DAMPING, TOL, out=out.data_ptr())
        return {"rank": out}
    engine.upload_vertex_data_ptr(state["init"].data_ptr())
    engine.setActive(*state["active"])
    stats = engine.run_schedule(state["schedule"])
    engine.download_vertex_data_ptr(out.data_ptr())
    if kind == "pagerank_app":
        return {"rank": out.view(torch.float32)[:, 0], "out_edges": out[:, 1]}
    return {"vertex_data": out, "iterations": stats.iterations}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its floating results in 64 bits
# ---------------------------------------------------------------------------
def work(case):
    """Each input read once and each output written once.  Edges are counted
    before duplicates go (they are 1 to 15 % of an R-MAT graph)."""
    if case["kind"] == "lanes":
        v = sum(_lane_sizes(case))
        e = 2 * v * case["edge_factor"]
        per_edge = 8 if case["what"] == "sssp" else 4
        flops = 2 * e * case["lanes"] if case["what"] == "ppr" else 0
        return {"bytes": e * per_edge + v * 4 * (1 + case["lanes"]), "flops": flops}
    v = case["vertices"]
    e = (2 if case["symmetric"] else 1) * v * case["edge_factor"]
    if case.get("islands"):
        v += case["islands"] * ISLAND_SIDE ** 2
        e += case["islands"] * 4 * ISLAND_SIDE * (ISLAND_SIDE - 1)
    if case["kind"] == "pagerank":
        return {"bytes": 4 * e + 8 * v, "flops": 2 * e}
    if case["kind"] == "pagerank_app":
        return {"bytes": 4 * e + 20 * v, "flops": 2 * e}
    if case["kind"] == "app":  # the edge list itself comes in
        return {"bytes": (12 if case["program"] == "sssp" else 8) * e + 8 * v, "flops": 0}
    per_edge = 8 if case["kind"] == "sssp" else 4
    return {"bytes": per_edge * e + 12 * v, "flops": 0}


def exact(case, seed):
    if case["kind"] == "pagerank":
        src, dst, n = _case_edges(case, seed)
        return {"rank": _power_iteration(src, dst, n, None)[:, 0]}
    if case["kind"] == "lanes" and case["what"] == "ppr":
        graphs, ids = _lane_graphs(case, seed)
        src, dst, seeds, base = [], [], [], 0
        for (v, s, d), row in zip(graphs, ids):
            src.append(s.long() + base)
            dst.append(d.long() + base)
            seeds.append(torch.from_numpy(row.astype(np.int64)).to(DEVICE) + base)
            base += v
        return {"rank": _power_iteration(torch.cat(src), torch.cat(dst), base,
                                         torch.stack(seeds))}
    return None  # whole numbers, or (pagerank_app) decided by 32-bit thresholds


def _power_iteration(src, dst, n, seeds):
    """PageRank columns r' = (1 - d) start + d * (sum over in-edges of r / out-degree)
    from r = start, until the largest column's L1 step is at most TOL.  start:
    1 / n everywhere, or (seeds [graphs][lanes]) 1 at each lane's seeds."""
    deg = torch.bincount(src, minlength=n).double()
    inv = torch.where(deg > 0, 1.0 / deg, torch.zeros_like(deg)).view(n, 1)
    if seeds is None:
        start = torch.full((n, 1), 1.0 / n, dtype=torch.float64, device=DEVICE)
    else:
        lanes = seeds.shape[1]
        start = torch.zeros((n, lanes), dtype=torch.float64, device=DEVICE)
        lane = torch.arange(lanes, device=DEVICE).expand_as(seeds)
        start[seeds.reshape(-1), lane.reshape(-1)] = 1.0
    rank, step = start, max(1, (1 << 28) // start.shape[1])
    for _ in range(1000):
        contrib, total = rank * inv, torch.zeros_like(rank)
        for a in range(0, src.shape[0], step):
            total.index_add_(0, dst[a:a + step], contrib[src[a:a + step]])
        new = (1.0 - DAMPING) * start + DAMPING * total
        residual = float((new - rank).abs().sum(0).max())
        rank = new
        if residual <= TOL:
            break
    return rank
