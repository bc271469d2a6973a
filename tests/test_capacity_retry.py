"""Queries that overflow their row pool and run again with a larger one (a small memory budget,
weights so alike that little is pruned), in a batch and at a server that has more queries
queued than slots: every answer is the one of an engine with room for all.  In a child process,
so that a server which stops answering ends as a failure."""
import json
import subprocess
import sys

import pytest

import gst_b200 as G
from conftest import PKG

pytestmark = pytest.mark.gpu

CHILD = """
import json, sys
sys.path.insert(0, sys.argv[1])
import gst_b200 as G
wmax, n, slots, how = int(sys.argv[2]), int(sys.argv[3]), int(sys.argv[4]), sys.argv[5]
g = G.synth_rmat(400_000, 700_000, 77, wmax=wmax)
grp = G.synth_groups_uniform(g.V, 300, 1, 3, 78)
qs = G.synth_queries(grp.n_groups, n, 7, 79)
eng = G.Engine(0, max_batch=slots, mem_budget_bytes=2 << 30, verbose=1)
dg = eng.graph(g, grp)
if how == "server":
    sv = dg.server()
    got = [sv.wait(t) for t in [sv.submit(q) for q in qs]]
    sv.close()
else:
    got = dg.solve_batch(qs, [None] * n)
print(json.dumps([(a.status, a.cost) for a in got]))
dg.close()
eng.close()
"""


@pytest.mark.parametrize("wmax", [1, 3])
def test_overflowing_queries_finish_with_their_optima(wmax):
    g = G.synth_rmat(400_000, 700_000, 77, wmax=wmax)
    grp = G.synth_groups_uniform(g.V, 300, 1, 3, 78)
    qs = G.synth_queries(grp.n_groups, 64, 7, 79)
    eng = G.Engine(0, batch_search=0)
    try:
        dg = eng.graph(g, grp)
        want = [(a.status, a.cost) for a in dg.solve_batch(qs, [None] * len(qs))]
        dg.close()
    finally:
        eng.close()
    for n, slots, how in [(40, 4, "server"), (64, 16, "server"), (40, 4, "batch")]:
        r = subprocess.run([sys.executable, "-c", CHILD, PKG, str(wmax), str(n), str(slots), how], capture_output=True,
                           text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
        assert r.stderr.count("[gst retry]") > 0, how
        assert [tuple(x) for x in json.loads(r.stdout)] == want[:n], (n, slots, how)
