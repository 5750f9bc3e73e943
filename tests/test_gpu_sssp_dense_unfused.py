"""Host-driven SSSP on dense graphs, where the threads of a step lower a vertex together: with
the strategies that relax whole lists a step queues a vertex once, so the queue holds them."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import (UDF, VUDF, GraphT, HostGraph, PriorityQueue, SimpleGPUSchedule as T, VertexData,
                                edgeset_apply, sssp, sssp_multi, vertexset_apply)

pytestmark = pytest.mark.gpu
LB = T.load_balancing_type


def dense(n, wmax):
    u, v = np.divmod(np.arange(n * n), n)
    return HostGraph.from_edges(n, u[u != v], v[u != v], np.random.default_rng(n).integers(1, wmax + 1, n * (n - 1)))


@pytest.mark.parametrize("n", [10, 33, 34, 400, 1100])  # lists of 9 edges and more
@pytest.mark.parametrize("wmax,delta", [(255, 32), (255, 2000), (100000, 3000)])
def test_distances_and_advances(n, wmax, delta):
    hg = dense(n, wmax)
    g = GraphT(hg)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    ref, adv = oracle.sssp_dijkstra(off, dst, w, 0), oracle.sssp_delta_gpu(off, dst, w, 0, delta)[1]
    for lb in (LB.VERTEX_BASED, LB.WM, LB.TWCE, LB.ETWC, LB.TWC):
        for cta in (128, 512):
            s = T().configLoadBalancing(lb)
            s.cta_size = cta
            d, st = sssp(g, 0, delta, s, fuse=False)
            np.testing.assert_array_equal(d, ref)
            assert st["bucket_advances"] == adv
    each = np.minimum(ref, oracle.sssp_dijkstra(off, dst, w, n - 1))
    np.testing.assert_array_equal(sssp_multi(g, np.array([0, n - 1], np.int32), delta,
                                             T().configLoadBalancing(LB.TWCE), False)[0], each)
    g.close()


@pytest.mark.parametrize("lb", [LB.VERTEX_BASED, LB.TWC, LB.TWCE])
def test_through_operators(lb):
    import torch
    hg = dense(400, 255)
    g = GraphT(hg)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    for src, delta in ((0, 32), (7, 2000)):
        sp = torch.empty(400, dtype=torch.int32, device="cuda")
        pq = PriorityQueue(g, sp, 0, delta, src)
        vertexset_apply(g, VUDF.SSSP_RESET, VertexData(dist=sp, src=src))
        while not pq.finished():
            edgeset_apply(T().configLoadBalancing(lb)).from_(pq.dequeue()).apply_priority(g, UDF.SSSP_RELAX, pq)
        pq.close()
        np.testing.assert_array_equal(sp.cpu().numpy(), oracle.sssp_dijkstra(off, dst, w, src))
    g.close()
