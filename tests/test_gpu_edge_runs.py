"""EDGE_ONLY PageRank pulls whose edges are summed in runs: block sizes that give 1, 2, 255,
256 and 257 buckets and more than the stable bucketing takes (1,024), edge counts around its
tile of 8,192 and around a warp's 128, a hub longer than a tile, and the unblocked walk."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, SimpleGPUSchedule as T, pagerank
from tests.conftest import rel_l1

pytestmark = pytest.mark.gpu
TOL = 1e-6  # fp32 ranks against FP64, as for every PageRank schedule


def schedule(block):
    s = T().configDirection(T.direction_type.PULL)
    if block:
        return s.configLoadBalancing(T.load_balancing_type.EDGE_ONLY, T.edge_blocking_type.BLOCKED, block)
    return s.configLoadBalancing(T.load_balancing_type.EDGE_ONLY)


def graph(vertices, edges, hub):
    """About `edges` random distinct edges, and one vertex with `hub` in-edges."""
    rng = np.random.default_rng(edges)
    key = np.unique(rng.integers(0, vertices * vertices, 2 * edges + 64))
    key = rng.permutation(key[key // vertices != key % vertices])[:edges]
    u, v = key // vertices, key % vertices
    if hub:
        h = np.arange(1, hub + 1)
        u, v = np.concatenate([u, h]), np.concatenate([v, np.zeros(hub, dtype=np.int64)])
    return HostGraph.from_edges(vertices, u, v)


@pytest.mark.parametrize("vertices,edges,hub", [(300, 31, 0), (300, 127, 0), (300, 129, 0), (2570, 8191, 0),
                                                (2570, 8192, 0), (2570, 8193, 0), (20000, 50000, 12000)])
def test_ranks(vertices, edges, hub):
    hg = graph(vertices, edges, hub)
    ref = oracle.pagerank(np.array(hg.offsets), np.array(hg.dst), 10, float(np.float32(0.85)))
    g = GraphT(hg)
    V = hg.num_vertices
    for buckets in (0, 1, 2, 255, 256, 257):
        block = -(-V // buckets) if buckets else 0
        r, _ = pagerank(g, 10, 0.85, schedule(block))
        assert rel_l1(r, ref) <= TOL, (buckets, rel_l1(r, ref))
    if not hub:
        r, _ = pagerank(g, 10, 0.85, schedule(2))  # 2,570 vertices: 1,285 buckets
        assert rel_l1(r, ref) <= TOL, rel_l1(r, ref)
    g.close()
