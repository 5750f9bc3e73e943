"""SSSP with a thread per vertex where every list is a hub's: the vertices of a step lower each
other's targets together, and the queue, of six entries a vertex, must hold what they find."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, SimpleGPUSchedule as T, sssp

pytestmark = pytest.mark.gpu
LB = T.load_balancing_type


@pytest.mark.parametrize("n", [1026, 1100, 1600])  # hubs from 1,025 edges on
@pytest.mark.parametrize("wmax,delta", [(255, 2000), (255, 64), (1000000, 1 << 21)])
def test_complete_graphs(n, wmax, delta):
    u, v = np.divmod(np.arange(n * n), n)
    u, v = u[u != v], v[u != v]
    hg = HostGraph.from_edges(n, u, v, np.random.default_rng(n).integers(1, wmax + 1, len(u)))
    g = GraphT(hg)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    ref = oracle.sssp_dijkstra(off, dst, w, 0)
    for cta in (128, 512):
        s = T().configLoadBalancing(LB.VERTEX_BASED)
        s.cta_size = cta
        np.testing.assert_array_equal(sssp(g, 0, delta, s, fuse=True)[0], ref)
    g.close()


def test_hubs_of_a_few():
    """Five centres that share their leaves: the step after the source's has five hubs in it."""
    leaves = np.arange(6, 20006)
    u = np.concatenate([np.zeros(5, np.int64), np.repeat(np.arange(1, 6), len(leaves))])
    v = np.concatenate([np.arange(1, 6), np.tile(leaves, 5)])
    hg = HostGraph.from_edges(20006, u, v, np.random.default_rng(2).integers(1, 256, len(u)), symmetrize=True)
    g = GraphT(hg, symmetric=True)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    for delta in (32, 2000):
        d = sssp(g, 0, delta, T().configLoadBalancing(LB.VERTEX_BASED), fuse=True)[0]
        np.testing.assert_array_equal(d, oracle.sssp_dijkstra(off, dst, w, 0))
    g.close()
