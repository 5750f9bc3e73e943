"""The one-CTA sessions of the fused SSSP loop on graphs of short lists (largest out-degree
at most 32): distances equal Dijkstra's and the bucket advances the reference rule's, where
the session's lists stay small, where they overflow into the queues and piles in global
memory, and on both sides of the degree limit."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import (BatchPlan, GraphT, HostGraph, SimpleGPUSchedule as T, sssp, sssp_multi)

pytestmark = pytest.mark.gpu
LB = T.load_balancing_type


def wheel(spokes, rng):
    """A ring of hubs, each with `spokes` leaves around it and back edges: many equal buckets
    and frontiers wider than the session's lists."""
    hubs = 400
    u, v = [], []
    for h in range(hubs):
        u += [h, (h + 1) % hubs]
        v += [(h + 1) % hubs, h]
        leaves = hubs + h * spokes + np.arange(spokes)
        u += [h] * spokes + leaves.tolist()
        v += leaves.tolist() + [(h + 7) % hubs] * spokes
    n = hubs + hubs * spokes
    return HostGraph.from_edges(n, u, v, rng.integers(1, 60, len(u)))


GRAPHS = {
    "line": lambda rng: HostGraph.grid(1, 3000),
    "grid": lambda rng: HostGraph.grid(97, 131),
    "unit": lambda rng: HostGraph.grid(120, 90, wmin=1, wmax=1),      # a bucket is a whole wavefront
    "heavy": lambda rng: HostGraph.grid(60, 60, wmin=1, wmax=100000),  # most parks are high
    "fan": lambda rng: wheel(28, rng),  # out-degree 30
    "fan33": lambda rng: wheel(33, rng),  # above the limit: the other path
}


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("delta", [1, 7, 128, 100000])
def test_distances_and_advances(name, delta):
    rng = np.random.default_rng(7)
    hg = GRAPHS[name](rng)
    g = GraphT(hg)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    for src, cta in ((0, 512), (hg.num_vertices - 1, 64)):
        sc = T().configLoadBalancing(LB.VERTEX_BASED)
        sc.cta_size = cta
        d, st = sssp(g, src, delta, sc, fuse=True)
        np.testing.assert_array_equal(d, oracle.sssp_dijkstra(off, dst, w, src))
        assert st["bucket_advances"] == oracle.sssp_delta_gpu(off, dst, w, src, delta)[1]
    g.close()


def test_multi_source_plan_on_a_mesh():
    import torch
    hg = HostGraph.grid(80, 75)
    g = GraphT(hg)
    srcs = hg.pick_sources(5)
    ref, _ = sssp_multi(g, srcs, 64)
    out = torch.empty(hg.num_vertices, dtype=torch.int32, device="cuda")
    plan = BatchPlan(g, "sssp_multi", srcs, out, delta=64)
    for _ in range(2):
        plan.run()
        np.testing.assert_array_equal(out.cpu().numpy(), ref)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    each = np.stack([oracle.sssp_dijkstra(off, dst, w, int(s)) for s in srcs])
    np.testing.assert_array_equal(ref, each.min(0))
    g.close()
