"""Pulled BFS levels with in-lists that the whole CTA walks: lists just below, at and above the
length from which they are set aside, with the frontier's vertex first, last or missing in
them, and more of them than a CTA sets aside."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, HybridGPUSchedule, bfs, default_schedule

pytestmark = pytest.mark.gpu


def fans(length, count):
    """A chain 0 -> 1 -> 2; `count` vertices with in-lists of `length` strays (never reached), and of
    those one in three with vertex 1 in front of the list, one in three with it at the end."""
    strays = 3 + count + np.arange(length)
    u, v = [np.array([0, 1])], [np.array([1, 2])]
    for i in range(count):
        t = 3 + i
        if i % 3 == 0:  # in-lists are sorted by id: vertex 1 comes first
            u.append(np.array([1])), v.append(np.array([t]))
        u.append(strays), v.append(np.full(length, t))
    n = 3 + count + length + 1
    u.append(np.array([1])), v.append(np.array([n - 1]))  # the last id, reached at depth 2
    for i in range(count):
        if i % 3 == 1:
            u.append(np.array([n - 1])), v.append(np.array([3 + i]))
    u, v = np.concatenate(u), np.concatenate(v)
    return HostGraph.from_edges(n, u, v)


@pytest.mark.parametrize("length", [507, 508, 511, 512, 513, 2048, 2049, 9000])
def test_set_aside_lists(length):
    power = default_schedule("bfs", power=True)[0]
    pull = HybridGPUSchedule(power.s1, power.s2).configThreshold(0.0)
    for count in (5, 700 if length < 2049 else 40):
        hg = fans(length, count)
        g = GraphT(hg)
        off, dst = np.array(hg.offsets), np.array(hg.dst)
        ref = oracle.bfs(off, dst, 0)
        assert ref.max() == 3 and (ref < 0).sum() >= length
        for s in (pull, power):
            depth, parent, st = bfs(g, 0, s, True, with_parent=True)
            np.testing.assert_array_equal(depth, ref)
            for v in np.nonzero(ref > 0)[0]:
                p = parent[v]
                assert ref[p] == ref[v] - 1 and v in dst[off[p]:off[p + 1]]
        g.close()
