"""SSSP where many threads lower one vertex in the same step (dense graphs, parallel edges):
near and far improvements of a vertex come in any order, and a pile still lists it once, so
its V entries suffice.  Distances equal Dijkstra's and the bucket advances the reference
rule's, for every fused strategy and many sources."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import BatchPlan, GraphT, HostGraph, SimpleGPUSchedule as T, sssp, sssp_multi

pytestmark = pytest.mark.gpu
LB = T.load_balancing_type


def complete(n, wmax):
    u, v = np.divmod(np.arange(n * n), n)
    u, v = u[u != v], v[u != v]
    return HostGraph.from_edges(n, u, v, np.random.default_rng(n).integers(1, wmax + 1, len(u)))


def random_dense(n, degree, wmax):
    rng = np.random.default_rng(n + degree)
    u = np.repeat(np.arange(n), degree)
    return HostGraph.from_edges(n, u, rng.integers(0, n, len(u)), rng.integers(1, wmax + 1, len(u)))


def parallel_edges(heavy, light):
    """Two vertices, 40 edges each way, heavy and light in turn."""
    w = np.tile(np.array([heavy, light], np.int32), 40)
    return HostGraph.from_csr(np.array([0, 40, 80], np.int32), np.repeat(np.array([1, 0], np.int32), 40), w)


GRAPHS = {f"K{n}_{w}": (lambda n=n, w=w: complete(n, w)) for n in (40, 64, 128, 400) for w in (255, 1000)}
GRAPHS.update({f"random{n}_{d}_{w}": (lambda n=n, d=d, w=w: random_dense(n, d, w))
               for n, d in ((100, 50), (300, 40), (1000, 200)) for w in (255, 1000)})
GRAPHS["parallel_low"] = lambda: parallel_edges(300, 5)
GRAPHS["parallel_high"] = lambda: parallel_edges(100000, 200)


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("delta", [32, 128])
def test_distances_and_advances(name, delta):
    hg = GRAPHS[name]()
    g = GraphT(hg)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    assert np.diff(off).max() > 32  # above the mesh sessions' limit
    ref, adv = oracle.sssp_dijkstra(off, dst, w, 0), oracle.sssp_delta_gpu(off, dst, w, 0, delta)[1]
    for lb in (LB.VERTEX_BASED, LB.WM, LB.TWCE, LB.CM):
        d, st = sssp(g, 0, delta, T().configLoadBalancing(lb), fuse=True)
        np.testing.assert_array_equal(d, ref)
        assert st["bucket_advances"] == adv
    srcs = np.unique([0, hg.num_vertices // 2, hg.num_vertices - 1]).astype(np.int32)
    each = np.stack([oracle.sssp_dijkstra(off, dst, w, int(s)) for s in srcs]).min(0)
    np.testing.assert_array_equal(sssp_multi(g, srcs, delta)[0], each)
    g.close()


def test_multi_source_plan():
    import torch
    hg = complete(200, 255)
    g = GraphT(hg)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    srcs = np.array([3, 77, 150], np.int32)
    out = torch.empty(200, dtype=torch.int32, device="cuda")
    plan = BatchPlan(g, "sssp_multi", srcs, out, delta=32)
    ref = np.stack([oracle.sssp_dijkstra(off, dst, w, int(s)) for s in srcs]).min(0)
    for _ in range(3):
        plan.run()
        np.testing.assert_array_equal(out.cpu().numpy(), ref)
    g.close()
