"""Hop-bounded shared searches whose last rounds pull at the members and their neighbours:
every bound D the shared search takes (1..8), alone and in a batch, on graphs whose groups
overlap (states of height 0 over several groups), against the oracle."""
import numpy as np
import pytest

import gst_b200 as G
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("V,m,smax,wmax", [(60, 150, 20, 5), (900, 4000, 4, 100), (2500, 5000, 60, 1 << 16)])
def test_pulled_rounds_keep_the_optimum(engine, D, V, m, smax, wmax):
    g = G.synth_rmat(V, m, 7 + V, wmax=wmax)
    grp = G.synth_groups_uniform(g.V, 40, 1, smax, 8)
    rng = np.random.default_rng(9 + D)
    qs = [rng.choice(40, size=int(k), replace=False).astype(np.int32) for k in (1, 2, 3, 4, 5, 5, 6)]
    dg = engine.graph(g, grp)
    try:
        got = dg.solve_batch(qs, [D] * len(qs))
        for q, a in zip(qs, got):
            want = O.gst_hop(g, grp, q, D)["cost"]
            for r in (a, dg.solve(q, D)):
                assert (r.cost if r.ok else -1) == want, (q, D)
                if r.ok:
                    assert G.verify_tree(g, grp, q, D, r.cost, r.edges, r.root) == 0
    finally:
        dg.close()
