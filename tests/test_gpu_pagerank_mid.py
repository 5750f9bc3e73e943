"""Static pull PageRank where the middle class (in-degrees 31 to 4,094, a warp each) is empty, a
part of a block, a block and one more, or just past one, two and five vertices a warp of the GPU."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, SimpleGPUSchedule as T, pagerank
from tests.conftest import rel_l1

pytestmark = pytest.mark.gpu
TOL = 1e-6  # as for every static pull
WARPS = 152 * 64


@pytest.mark.parametrize("mid", [0, 1, 7, 8, 9, WARPS - 1, WARPS, 2 * WARPS - 1, 2 * WARPS + 3, 5 * WARPS + 7])
@pytest.mark.parametrize("hub", [False, True])
def test_middle_class(mid, hub):
    rng = np.random.default_rng(mid)
    n = mid + 9000
    u = [np.arange(n)]                       # a ring, so that every vertex has an out-edge
    v = [(np.arange(n) + 1) % n]
    u.append((np.repeat(np.arange(mid), 40) * 7 + 13 * np.tile(np.arange(40), mid)) % n)
    v.append(np.repeat(np.arange(mid), 40))  # 39 or 40 in-edges, and the ring's
    if hub:
        u.append(np.arange(n)), v.append(np.full(n, n - 1))
    hg = HostGraph.from_edges(n, np.concatenate(u), np.concatenate(v))
    g = GraphT(hg)
    off, dst = np.array(hg.offsets), np.array(hg.dst)
    indeg = np.bincount(dst, minlength=n)
    assert ((indeg >= 31) & (indeg < 4095)).sum() == mid
    s = T().configDirection(T.direction_type.PULL).configLoadBalancing(T.load_balancing_type.TWC)
    r, _ = pagerank(g, 12, 0.85, s)
    assert rel_l1(r, oracle.pagerank(off, dst, 12, float(np.float32(0.85)))) <= TOL
    np.testing.assert_array_equal(r, pagerank(g, 12, 0.85, s)[0])
    g.close()
