"""BC in one persistent kernel (a simple push schedule with fusion on): every strategy the fused
loops have, on skewed, mesh and directed graphs, a chain of as many levels as vertices, a source
without edges, and a hub that goes through the hub list; against the FP64 oracle, and the
counters of the unfused run."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, SimpleGPUSchedule as T, bc
from tests.conftest import rel_l1

pytestmark = pytest.mark.gpu
LB = T.load_balancing_type
TOL = 1e-6  # fp32 dependencies against FP64, as for every BC schedule


def star():
    leaves = np.arange(1, 30001)  # more than 8 CTA widths of 512
    ring = np.arange(1, 30000, 7)
    return HostGraph.from_edges(30001, np.concatenate([np.zeros(30000, np.int64), ring]),
                                np.concatenate([leaves, ring + 1]), symmetrize=True)


GRAPHS = {
    "rmat12": lambda: HostGraph.rmat(12, 16, symmetrize=True),
    "rmat11_directed": lambda: HostGraph.rmat(11, 8),
    "grid": lambda: HostGraph.grid(37, 29),
    "chain": lambda: HostGraph.grid(1, 700),
    "star": star,
    "isolated": lambda: HostGraph.from_edges(5, [1, 2], [2, 3], symmetrize=True),
}


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("lb", [LB.TWCE, LB.VERTEX_BASED, LB.WM, LB.CM])
def test_dependencies(name, lb):
    hg = GRAPHS[name]()
    g = GraphT(hg, symmetric=name not in ("rmat11_directed",))
    off, dst = np.array(hg.offsets), np.array(hg.dst)
    for src in {0, int(np.argmax(np.diff(off))), hg.num_vertices - 1}:
        s = T().configLoadBalancing(lb)
        dep, st = bc(g, src, s, True)
        ref, plain = bc(g, src, s, False)
        assert rel_l1(dep, oracle.bc(off, dst, src)) <= TOL
        np.testing.assert_allclose(dep, ref, rtol=1e-6, atol=1e-6 * max(1.0, float(np.abs(ref).max())))
        for key in ("iterations", "push_iterations", "vertices_reached", "edges_traversed"):
            assert st[key] == plain[key], (key, st[key], plain[key])
        assert st["fused"] == 1
    g.close()
