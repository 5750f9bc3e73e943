"""Host-driven SSSP on dense graphs, where the threads of a step lower a vertex together: with
the strategies that relax whole lists a step queues a vertex once, so the queue holds them."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, SimpleGPUSchedule as T, sssp, sssp_multi

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
