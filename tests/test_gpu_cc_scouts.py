"""Fused CC where its second sampling round is split into scouts and the rest (262,144
vertices and more) and just below: labels are the minimum id of each component."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, cc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vertices", [262143, 262144, 262145, 300007])
@pytest.mark.parametrize("symmetrize", [True, False])
def test_labels_around_the_split(vertices, symmetrize):
    rng = np.random.default_rng(vertices)
    # sparse random edges: many components besides the giant one, and isolated vertices
    m = vertices * 3 // 4
    hg = HostGraph.from_edges(vertices, rng.integers(0, vertices, m), rng.integers(0, vertices, m),
                              symmetrize=symmetrize)
    g = GraphT(hg, symmetric=symmetrize)
    labels, _ = cc(g, fuse=True)
    np.testing.assert_array_equal(labels, oracle.cc(np.array(hg.offsets), np.array(hg.dst)))
    g.close()
