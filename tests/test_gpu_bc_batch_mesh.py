"""Batched BC where a level holds a few items: most warps find none left, on lines, grids and a
small skewed graph whose hubs are long items; against the FP64 oracle, twice on the same state."""
import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import BatchPlan, GraphT, HostGraph, bc_batch, set_batch_tuning
from tests.conftest import rel_l1

pytestmark = pytest.mark.gpu
TOL = 1e-6  # fp32 dependencies against FP64, as for every BC schedule

GRAPHS = {
    "line": lambda: HostGraph.grid(1, 900),
    "grid": lambda: HostGraph.grid(41, 29),
    "rmat9": lambda: HostGraph.rmat(9, 40, symmetrize=True),  # lists above and below a light item
}


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("nsrc", [1, 64])
def test_few_items(name, nsrc):
    import torch
    hg = GRAPHS[name]()
    g = GraphT(hg, symmetric=True)
    off, dst = np.array(hg.offsets), np.array(hg.dst)
    srcs = hg.pick_sources(nsrc)
    ref = np.stack([oracle.bc(off, dst, int(s)) for s in srcs])
    out = torch.empty((nsrc, hg.num_vertices), dtype=torch.float32, device="cuda")
    plan = BatchPlan(g, "bc", srcs, out)
    for _ in range(2):
        rows, _ = bc_batch(g, srcs)
        plan.run()
        for s in range(nsrc):
            assert rel_l1(rows[s], ref[s]) <= TOL
            assert rel_l1(out[s].cpu().numpy(), ref[s]) <= TOL
    g.close()


@pytest.mark.parametrize("chunk", [32, 64, 128, 256])
def test_item_sizes(chunk):
    """The tuning's chunk bounds every work item, also where it is below a light item's size."""
    hg = HostGraph.rmat(9, 40, symmetrize=True)
    g = GraphT(hg, symmetric=True)
    off, dst = np.array(hg.offsets), np.array(hg.dst)
    srcs = hg.pick_sources(5)
    set_batch_tuning(g, "bc", chunk=chunk)
    rows, _ = bc_batch(g, srcs)
    for s, row in zip(srcs, rows):
        assert rel_l1(row, oracle.bc(off, dst, int(s))) <= TOL
    g.close()
