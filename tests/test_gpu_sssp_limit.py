"""A mesh session of the fused SSSP loop keeps to its time slice whatever the order of its
rounds: on a line of unit weights at delta 1 relaxes and advances take turns, and the loop's
wall-clock limit must be met then too.  The limit is read from the environment, in a child."""
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

import oracle
from easy_graphit_gb300 import GraphT, HostGraph, SimpleGPUSchedule as T, sssp
from easy_graphit_gb300 import _lib as L
from tests.conftest import ROOT

pytestmark = pytest.mark.gpu


def test_limit_is_met_where_relaxes_and_advances_take_turns():
    code = "import sys\nsys.path.insert(0, %r)\n" % str(ROOT) + textwrap.dedent("""
        import time
        from easy_graphit_gb300 import GraphT, HostGraph, SimpleGPUSchedule as T, sssp
        from easy_graphit_gb300 import _lib as L
        g = GraphT(HostGraph.grid(1, 3000000, wmin=1, wmax=1), symmetric=True)
        for _ in range(2):
            t0 = time.perf_counter()
            try:
                sssp(g, 0, 1, T(), True)
                print("NO_TIMEOUT")
            except L.GGError as e:
                print("STATUS", e.status, "SECONDS", time.perf_counter() - t0)
    """)
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, GG_LOOP_TIMEOUT_MS="20"),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    lines = r.stdout.split("\n")[:2]
    assert all(f"STATUS {L.GG_ERR_TIMEOUT}" in x for x in lines), r.stdout
    # the second call: 20 ms, a slice of 1 ms, and the copy of 3 M distances
    assert float(lines[1].split()[-1]) < 0.2, r.stdout


@pytest.mark.parametrize("delta", [1, 3])
def test_unit_line(delta):
    hg = HostGraph.grid(1, 20011, wmin=1, wmax=1)
    g = GraphT(hg, symmetric=True)
    off, dst, w = np.array(hg.offsets), np.array(hg.dst), np.array(hg.weights)
    d, st = sssp(g, 7, delta, T(), True)
    np.testing.assert_array_equal(d, np.abs(np.arange(20011) - 7))
    assert st["bucket_advances"] == oracle.sssp_delta_gpu(off, dst, w, 7, delta)[1]
    g.close()
