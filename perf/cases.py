"""Performance cases of the framework: what its users run, through its public Python API.

Every case is one call that a program makes on a graph it already holds on the GPU
(`GraphT`, and where it has one its `BatchPlan` or learned schedule): single-source BFS,
delta-stepping SSSP, PageRank, connected components and betweenness centrality, and the
batched forms with many sources in one call.  Graphs are the two families of the
framework's tests and benchmark: R-MAT (a/b/c/d 0.57/0.19/0.19/0.05, skewed degrees, a
handful of levels) and 4-neighbour grids (degree 4, thousands of small buckets).  They are
made on the GPU from the seed alone: sorted, deduplicated, without self-loops, int32
weights in [1, 255] (R-MAT) or [1, 1000] (grid).
"""
import numpy as np
import torch

from easy_graphit_gb300 import (BatchPlan, GraphT, LearnedGPUSchedule, Selector,
                                SimpleGPUSchedule, bc, bc_batch, bfs, bfs_batch, cc, default_schedule,
                                pagerank, sssp, sssp_batch)

LB = SimpleGPUSchedule.load_balancing_type
DIR = SimpleGPUSchedule.direction_type
DEVICE = "cuda"


def listed():
    return [
        # The smallest call: BFS on a graph of a thousand vertices with bfs.cpp's own schedule.  A
        # service that answers one query after another on small graphs pays launches and latency.
        {"name": "bfs_small", "app": "bfs", "graph": "rmat", "vertices": 1000, "degree": 16,
         "symmetric": True, "schedule": "default"},
        # One traversal of a large directed graph with the learned direction per level.
        {"name": "bfs_large", "app": "bfs", "graph": "rmat", "vertices": 4194304, "degree": 16,
         "symmetric": False, "schedule": "learned"},
        # sssp.cpp with its own schedule (thread per vertex, fused) on a mid-sized skewed graph.
        {"name": "sssp_rmat", "app": "sssp", "graph": "rmat", "vertices": 250007, "degree": 16,
         "symmetric": False, "schedule": "default", "delta": 32},
        # The same call on a road-like mesh: high diameter, many small buckets.
        {"name": "sssp_grid", "app": "sssp", "graph": "grid", "rows": 700, "cols": 501,
         "schedule": "default", "delta": 128},
        # pr.cpp with its own schedule (pull, edge-only, blocked) ...
        {"name": "pagerank_default", "app": "pagerank", "graph": "rmat", "vertices": 1000003, "degree": 15,
         "symmetric": False, "schedule": "default", "iters": 20},
        # ... and with the pull schedule that suits static graphs, at full size.
        {"name": "pagerank_pull", "app": "pagerank", "graph": "rmat", "vertices": 4194304, "degree": 16,
         "symmetric": False, "schedule": "pull_twc", "iters": 20},
        # Components of an undirected graph in one fused pass.
        {"name": "cc_fused", "app": "cc", "graph": "rmat", "vertices": 4194304, "degree": 16,
         "symmetric": True, "fuse": True},
        # bc.cpp with its own schedule: the operator-by-operator path, forward and backward sweeps.
        {"name": "bc_single", "app": "bc", "graph": "rmat", "vertices": 100003, "degree": 16,
         "symmetric": True, "schedule": "default"},
        # 64 BFS sources replayed from a captured plan: a service's steady state.
        {"name": "bfs_batch", "app": "bfs_batch", "graph": "rmat", "vertices": 1048576, "degree": 16,
         "symmetric": False, "sources": 64, "plan": True},
        # The benchmark's headline workload: 32 delta-stepping sources on a directed R-MAT 22.
        {"name": "sssp_batch", "app": "sssp_batch", "graph": "rmat", "vertices": 4194304, "degree": 16,
         "symmetric": False, "sources": 32, "delta": 32, "plan": False},
        # The batch on a mesh, where every source gets a loop of its own.
        {"name": "sssp_batch_grid", "app": "sssp_batch", "graph": "grid", "rows": 500, "cols": 501,
         "sources": 32, "delta": 32, "plan": False},
        # Betweenness centrality from 64 sources of an undirected graph.
        {"name": "bc_batch", "app": "bc_batch", "graph": "rmat", "vertices": 524287, "degree": 16,
         "symmetric": True, "sources": 64, "plan": False},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, odd ones among them."""
    app = rng.choice(["bfs", "bfs", "sssp", "sssp", "pagerank", "cc", "bc", "bfs_batch", "sssp_batch", "bc_batch"])
    most = {"bfs": 4194304, "sssp": 250007, "pagerank": 4194304, "cc": 4194304, "bc": 100003,
            "bfs_batch": 1048576, "sssp_batch": 4194304, "bc_batch": 524287}[app]
    case = {"app": app}
    if app in ("sssp", "sssp_batch") and rng.random() < 0.4:
        side = 700 if app == "sssp" else 500
        case.update(graph="grid", rows=_log_int(rng, 40, side), cols=_log_int(rng, 40, 501))
    else:
        case.update(graph="rmat", vertices=_log_int(rng, 1000, most), degree=rng.randint(5, 16),
                    symmetric=True if app in ("bc", "bc_batch") else rng.random() < 0.5)
    if app in ("sssp", "sssp_batch"):
        case["delta"] = rng.choice([32, 128])
    if app == "bfs":
        case["schedule"] = rng.choice(["default", "power_fused", "learned"])
    elif app == "sssp":
        case["schedule"] = rng.choice(["default", "twce_fused"])
    elif app == "pagerank":
        case["schedule"] = "pull_twc" if case["vertices"] > 1000003 else rng.choice(["default", "pull_twc"])
        case["iters"] = rng.randint(5, 20)
    elif app == "cc":
        case["fuse"] = True if case["vertices"] > 1000003 else rng.random() < 0.7
    elif app == "bc":
        case["schedule"] = rng.choice(["default", "power"])
    else:
        case["sources"] = rng.randint(1, 32 if app == "sssp_batch" else 64)
        case["plan"] = rng.random() < 0.5
    return case


# ------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _csr(vertices, key, w):
    """CSR of sorted keys u * vertices + v."""
    u = torch.div(key, vertices, rounding_mode="floor")
    dst = (key - u * vertices).to(torch.int32)
    off = torch.searchsorted(u, torch.arange(vertices + 1, device=DEVICE, dtype=torch.int64)).to(torch.int32)
    return off, dst, w


def _rmat(vertices, degree, symmetric, gen):
    """R-MAT edges over the covering power of two, folded onto `vertices` ids and permuted."""
    m, scale = vertices * degree, max(1, (vertices - 1).bit_length())
    u = torch.zeros(m, dtype=torch.int64, device=DEVICE)
    v = torch.zeros(m, dtype=torch.int64, device=DEVICE)
    for _ in range(scale):
        r = torch.rand(m, device=DEVICE, generator=gen)
        u = 2 * u + (r > 0.76)
        v = 2 * v + (((r > 0.57) & (r <= 0.76)) | (r > 0.95))
    perm = torch.randperm(vertices, device=DEVICE, generator=gen)
    u, v = perm[u % vertices], perm[v % vertices]
    keep = u != v
    u, v = u[keep], v[keep]
    if not symmetric:
        key = torch.unique(u * vertices + v)
        return _csr(vertices, key, torch.randint(1, 256, key.shape, device=DEVICE, generator=gen, dtype=torch.int32))
    pair = torch.unique(torch.minimum(u, v) * vertices + torch.maximum(u, v))
    w = torch.randint(1, 256, pair.shape, device=DEVICE, generator=gen, dtype=torch.int32)
    lo = torch.div(pair, vertices, rounding_mode="floor")
    key, order = torch.sort(torch.cat([pair, (pair - lo * vertices) * vertices + lo]))
    return _csr(vertices, key, torch.cat([w, w])[order].contiguous())


def _grid(rows, cols, gen):
    at = torch.arange(rows * cols, device=DEVICE, dtype=torch.int64).view(rows, cols)
    a = torch.cat([at[:, :-1].reshape(-1), at[:-1, :].reshape(-1)])
    b = torch.cat([at[:, 1:].reshape(-1), at[1:, :].reshape(-1)])
    n = rows * cols
    key = torch.sort(torch.cat([a * n + b, b * n + a])).values
    return _csr(n, key, torch.randint(1, 1001, key.shape, device=DEVICE, generator=gen, dtype=torch.int32))


def _inputs(case, seed):
    """(offsets, dst, weights, sources) of the case, on the GPU; sources as the programs pick them:
    the vertex of highest degree for one traversal, vertices with out-edges for a batch."""
    gen = _generator(seed)
    if case["graph"] == "grid":
        off, dst, w = _grid(case["rows"], case["cols"], gen)
    else:
        off, dst, w = _rmat(case["vertices"], case["degree"], case["symmetric"], gen)
    deg = off[1:] - off[:-1]
    if "sources" in case or case["graph"] == "grid":
        some = deg.nonzero().view(-1)
        src = some[torch.randint(some.numel(), (case.get("sources", 1),), device=DEVICE, generator=gen)]
    else:
        src = deg.argmax().view(1)
    return off, dst, w, src.to(torch.int32).cpu().numpy()


def _schedule(case):
    """(schedule, fuse) of the case's call."""
    app, kind = case["app"], case.get("schedule", "default")
    if kind == "power":
        return default_schedule(app, power=True)
    if kind == "power_fused":
        return default_schedule(app, power=True)[0], True
    if kind == "learned":
        return LearnedGPUSchedule(Selector.pretrained_fused_bfs()), True
    if kind == "twce_fused":
        return SimpleGPUSchedule().configLoadBalancing(LB.TWCE), True
    if kind == "pull_twc":
        return SimpleGPUSchedule().configDirection(DIR.PULL).configLoadBalancing(LB.TWC), False
    return None, None


def prepare(case, seed):
    off, dst, w, srcs = _inputs(case, seed)
    torch.cuda.synchronize()  # the graph copies the arrays on a stream of its own
    g = GraphT(offsets=off, dst=dst, weights=w, symmetric=case.get("symmetric", False))
    state = {"case": case, "g": g, "src": int(srcs[0]), "srcs": srcs}
    state["schedule"], state["fuse"] = _schedule(case)
    app = case["app"]
    if app.endswith("_batch"):
        dtype = torch.float32 if app == "bc_batch" else torch.int32
        state["out"] = torch.empty((len(srcs), g.num_vertices), dtype=dtype, device=DEVICE)
        if case["plan"]:
            state["plan"] = BatchPlan(g, app[:-6], srcs, state["out"], delta=case.get("delta", 32))
    return state


def run(state):
    case, g, sched, fuse = state["case"], state["g"], state["schedule"], state["fuse"]
    app = case["app"]
    if app == "bfs":
        return bfs(g, state["src"], sched, fuse)[0]
    if app == "sssp":
        return sssp(g, state["src"], case["delta"], sched, fuse)[0]
    if app == "pagerank":
        return pagerank(g, case["iters"], schedule=sched)[0]
    if app == "cc":
        return cc(g, fuse=case["fuse"])[0]
    if app == "bc":
        return bc(g, state["src"], sched, fuse)[0]
    if "plan" in state:
        state["plan"].run()
        return state["out"]
    if app == "bfs_batch":
        return bfs_batch(g, state["srcs"], out=state["out"])[0]
    if app == "sssp_batch":
        return sssp_batch(g, state["srcs"], case["delta"], out=state["out"])[0]
    return bc_batch(g, state["srcs"], out=state["out"])[0]


def work(case):
    """The graph read once (requested edges; repeated ones and self-loops drop out of the R-MAT) and
    the result written once; float operations of the sums over edges."""
    if case["graph"] == "grid":
        v = case["rows"] * case["cols"]
        e = 4 * v - 2 * (case["rows"] + case["cols"])
    else:
        v = case["vertices"]
        e = v * case["degree"] * (2 if case["symmetric"] else 1)
    app, k = case["app"], case.get("sources", 1)
    weights = 4 * e if app.startswith("sssp") else 0
    flops = {"pagerank": 2 * e * case.get("iters", 0) if app == "pagerank" else 0, "bc": 2 * e,
             "bc_batch": 2 * e * k}.get(app, 0)
    return {"bytes": 4 * e + weights + 4 * v + 4 * v * k, "flops": flops}


# ---------------------------------------------------- results in 64 bits
def _pagerank64(off, dst, iters):
    v = off.numel() - 1
    deg = (off[1:] - off[:-1]).to(torch.float64)
    src = torch.repeat_interleave(torch.arange(v, device=DEVICE), (off[1:] - off[:-1]).long())
    order = torch.argsort(dst, stable=True)
    src = src[order]
    counts = torch.bincount(dst.long(), minlength=v)
    damp = float(np.float32(0.85))
    rank = torch.full((v,), 1.0 / v, dtype=torch.float64, device=DEVICE)
    for _ in range(iters):
        share = (rank / deg)[src]
        rank = (1.0 - damp) / v + damp * torch.segment_reduce(share, "sum", lengths=counts, unsafe=True, initial=0.0)
    return rank


def _dependences64(off, dst, source):
    """Brandes dependencies of one source on a symmetric graph."""
    v = off.numel() - 1
    start, deg = off[:-1].long(), (off[1:] - off[:-1]).long()

    def edges_of(front):
        n = deg[front]
        u = torch.repeat_interleave(front, n)
        first = torch.repeat_interleave(torch.cumsum(n, 0) - n, n)
        k = torch.repeat_interleave(start[front], n) + torch.arange(u.numel(), device=DEVICE) - first
        return u, dst[k].long()

    depth = torch.full((v,), -1, dtype=torch.int64, device=DEVICE)
    sigma = torch.zeros(v, dtype=torch.float64, device=DEVICE)
    dep = torch.zeros(v, dtype=torch.float64, device=DEVICE)
    front = torch.tensor([source], device=DEVICE)
    depth[front], sigma[front] = 0, 1.0
    levels = []
    while front.numel():
        u, x = edges_of(front)
        new = depth[x] < 0
        u, x = u[new], x[new]
        levels.append((u, x))
        sigma.index_add_(0, x, sigma[u])
        front = torch.unique(x)
        depth[front] = len(levels)
    for u, x in reversed(levels):
        dep.index_add_(0, u, sigma[u] / sigma[x] * (1.0 + dep[x]))
    return dep


def exact(case, seed):
    """PageRank and BC in 64 bits; the other apps return whole numbers."""
    if case["app"] not in ("pagerank", "bc", "bc_batch"):
        return None
    off, dst, _, srcs = _inputs(case, seed)
    if case["app"] == "pagerank":
        return _pagerank64(off, dst, case["iters"])
    if case["app"] == "bc":
        return _dependences64(off, dst, int(srcs[0]))
    return torch.stack([_dependences64(off, dst, int(s)) for s in srcs])
