"""Hubs whose finds outgrow a CTA's stage in one step: appends go on to the queue or pile
directly.  BFS and SSSP on a star with a ring through its leaves and on an R-MAT graph, every
strategy, fused and not, at the smallest CTA, the default and the largest."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, SimpleGPUSchedule as T, bfs, sssp

pytestmark = pytest.mark.gpu
LB = T.load_balancing_type


def star():
    leaves = np.arange(1, 20001)
    ring = np.arange(1, 20000, 3)
    u, v = np.concatenate([np.zeros(20000, np.int64), ring]), np.concatenate([leaves, ring + 1])
    return HostGraph.from_edges(20001, u, v, np.random.default_rng(3).integers(1, 256, len(u)), symmetrize=True)


@pytest.mark.parametrize("name", ["star", "rmat14"])
@pytest.mark.parametrize("cta", [64, 512, 1024])
def test_depths_and_distances(name, cta):
    hg = star() if name == "star" else HostGraph.rmat(14, 16, symmetrize=True)
    g = GraphT(hg, symmetric=True)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    src = int(np.argmax(np.diff(off)))
    depth, dist = oracle.bfs(off, dst, src), {d: oracle.sssp_dijkstra(off, dst, w, src) for d in (32, 2000)}
    for lb in (LB.VERTEX_BASED, LB.WM, LB.TWCE, LB.CM, LB.ETWC, LB.TWC, LB.STRICT):
        s = T().configLoadBalancing(lb)
        s.cta_size = cta
        for fuse in (True, False):
            if fuse and lb in (LB.ETWC, LB.TWC, LB.STRICT):
                continue
            np.testing.assert_array_equal(bfs(g, src, s, fuse)[0], depth)
            for delta in (32, 2000):
                np.testing.assert_array_equal(sssp(g, src, delta, s, fuse)[0], dist[delta])
    g.close()
