"""TWCE slices on graphs whose longest list leaves them no, little or much work: lists of 1, 7,
8, 9, 31, 32, 33 and 700 edges, frontiers of one vertex and of many, pushed and pulled."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, SimpleGPUSchedule as T, bc, bfs, bfs_batch, sssp
from tests.conftest import rel_l1

pytestmark = pytest.mark.gpu
LB, DIR = T.load_balancing_type, T.direction_type


def fan(degree, spread):
    """Vertex i leads to the `degree` vertices after it, at steps of `spread`; directed."""
    n = 3000
    u = np.repeat(np.arange(n), degree)
    v = (u + 1 + spread * np.tile(np.arange(degree), n)) % n
    return HostGraph.from_edges(n, u, v, np.random.default_rng(degree).integers(1, 100, len(u)))


@pytest.mark.parametrize("degree", [1, 7, 8, 9, 31, 32, 33, 700])
def test_every_list_is_walked_whole(degree):
    hg = fan(degree, 3)
    g = GraphT(hg)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    assert np.diff(off).max() == degree
    depth, dist, ref = oracle.bfs(off, dst, 5), oracle.sssp_dijkstra(off, dst, w, 5), oracle.bc(off, dst, 5)
    for cta in (64, 512):
        for lb in (LB.TWCE, LB.ETWC):
            s = T().configLoadBalancing(lb)
            s.cta_size = cta
            for fuse in ((True, False) if lb == LB.TWCE else (False,)):
                np.testing.assert_array_equal(bfs(g, 5, s, fuse)[0], depth)
                if fuse:
                    np.testing.assert_array_equal(sssp(g, 5, 64, s, True)[0], dist)
                assert rel_l1(bc(g, 5, s, fuse)[0], ref) <= 1e-6
            p = T().configDirection(DIR.PULL).configLoadBalancing(lb)
            p.cta_size = cta
            np.testing.assert_array_equal(bfs(g, 5, p, False)[0], depth)
    srcs = np.array([5, 1700, 2999], np.int32)
    rows = bfs_batch(g, srcs)[0]
    for s, row in zip(srcs, rows):
        np.testing.assert_array_equal(row, oracle.bfs(off, dst, int(s)))
    g.close()
