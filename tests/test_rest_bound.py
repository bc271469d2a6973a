"""The rest bounds that limit the edges of a grow step and the states a merge keeps: the
bound of a group set is at most the optimum of the query over those groups (CPU, against
the oracle), and the engine keeps the optimum where the bounds bite (GPU): k from 1 to 8,
light and heavy weights, overlapping groups, with and without a hop bound."""
from itertools import permutations

import numpy as np
import pytest

import gst_b200 as G
import oracle as O
from test_shared_search_model import _bf, exact_hop


def rest_bound(vv, X):
    """max(largest group distance, half of the cheapest closed sequence through X)."""
    if len(X) < 2:
        return 0
    far = max(vv[a][b] for a in X for b in X if a != b)
    walk = min(sum(vv[p[i]][p[(i + 1) % len(p)]] for i in range(len(p))) for p in permutations(X))
    return max(far, (walk + 1) // 2)


@pytest.mark.parametrize("hop", [None, 2, 4])
@pytest.mark.parametrize("wmax", [3, 100])
def test_rest_bounds_never_exceed_the_optimum(hop, wmax):
    for seed in range(3):
        g = G.synth_rmat(300, 900, 50 + seed, wmax=wmax)
        grp = G.synth_groups_uniform(g.V, 20, 1, 6, 60 + seed)
        for q in G.synth_queries(grp.n_groups, 4, 5, 70 + seed):
            sets = [grp.members[grp.grp_ptr[i]:grp.grp_ptr[i + 1]] for i in q]
            d = _bf(g.beg_pos, g.adj, g.weight, sets) if hop is None else \
                exact_hop(g.beg_pos, g.adj, g.weight, sets, hop)[hop]
            vv = [[int(d[j][sets[i]].min()) for j in range(5)] for i in range(5)]
            for bits in range(1, 32):
                X = [i for i in range(5) if bits >> i & 1]
                o = O.gst_nonhop(g, grp, q[X]) if hop is None else O.gst_hop(g, grp, q[X], hop)
                assert o["cost"] < 0 or rest_bound(vv, X) <= o["cost"], (q, X)


@pytest.mark.gpu
@pytest.mark.parametrize("k,hop", [(1, None), (2, None), (2, 3), (5, 2), (7, None), (7, 3), (8, None)])
@pytest.mark.parametrize("wmax", [2, 100, 1 << 20, 1 << 24])
def test_engine_keeps_the_optimum(engine, k, hop, wmax):
    g = G.synth_rmat(700, 3000, 90 + k, wmax=wmax)
    grp = G.synth_groups_uniform(g.V, 30, 1, 40, 91)
    dg = engine.graph(g, grp)
    try:
        qs = G.synth_queries(grp.n_groups, 4, k, 92)
        for q, a in zip(qs, dg.solve_batch(qs, [hop] * len(qs))):
            o = O.gst_nonhop(g, grp, q) if hop is None else O.gst_hop(g, grp, q, hop)
            assert (a.cost if a.ok else -1) == o["cost"], (q, hop)
            if a.ok:
                assert G.verify_tree(g, grp, q, -1 if hop is None else hop, a.cost, a.edges, a.root) == 0
    finally:
        dg.close()
