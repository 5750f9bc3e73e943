"""Fused BFS on meshes: thousands of levels of a few vertices, where what a level pays beside
its edges decides.  Depths for every fused strategy, the hybrid rule and the learned direction,
and the cost of a level."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import (GraphT, HostGraph, HybridGPUSchedule, LearnedGPUSchedule, Selector,
                                SimpleGPUSchedule as T, bfs, bfs_multi, default_schedule)

pytestmark = pytest.mark.gpu
LB = T.load_balancing_type


def schedules():
    power = default_schedule("bfs", power=True)[0]
    out = {lb.name: T().configLoadBalancing(lb) for lb in (LB.TWCE, LB.VERTEX_BASED, LB.WM, LB.CM)}
    out["hybrid"] = power
    out["pull"] = HybridGPUSchedule(power.s1, power.s2).configThreshold(0.0)
    out["learned"] = LearnedGPUSchedule(Selector.pretrained_fused_bfs())
    small = T().configLoadBalancing(LB.TWCE)
    small.cta_size = 64
    out["TWCE_64"] = small
    return out


@pytest.mark.parametrize("rows,cols", [(1, 1500), (97, 131), (200, 200)])
def test_depths(rows, cols):
    hg = HostGraph.grid(rows, cols)
    g = GraphT(hg, symmetric=True)
    off, dst = np.array(hg.offsets), np.array(hg.dst)
    for src in (0, rows * cols // 2):
        ref = oracle.bfs(off, dst, src)
        for name, s in schedules().items():
            depth, _, st = bfs(g, src, s, True)
            np.testing.assert_array_equal(depth, ref, err_msg=name)
            assert st["iterations"] == ref.max() + 1, name
    srcs = np.array([0, rows * cols // 3, rows * cols - 1], np.int32)
    each = np.stack([oracle.bfs(off, dst, int(s)) for s in srcs]).min(0)
    np.testing.assert_array_equal(bfs_multi(g, srcs)[0], each)
    g.close()


def test_cost_of_a_level():
    """398 levels of up to 200 vertices: 5.5 us each, 11.4 where every warp reads the control words."""
    g = GraphT(HostGraph.grid(200, 200), symmetric=True)
    s = T().configLoadBalancing(LB.TWCE)
    runs = [bfs(g, 0, s, True)[2] for _ in range(8)]
    assert min(st["loop_ms"] for st in runs) / runs[0]["iterations"] < 8.5e-3
    g.close()
