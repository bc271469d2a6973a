"""The scan of four vertices a thread (graphs of 2,000,000 vertices on): vertex counts that leave 1, 2
and 3 vertices in the last quad, 1 to 8 mask words a vertex, pushing and pulling rounds of every
hop bound, one and two edge classes, against queries that search on their own.  And the bounds
D = 6 and 7 on small graphs, against the oracle."""
import numpy as np
import pytest

import gst_b200 as G
import oracle as O

pytestmark = pytest.mark.gpu


def _graph(V, m, seed):
    """A random tree and m more edges, weights 1..50."""
    rng = np.random.default_rng(seed)
    u = np.concatenate([np.arange(1, V), rng.integers(0, V, m)])
    v = np.concatenate([(np.arange(1, V) * rng.random(V - 1)).astype(np.int64), rng.integers(0, V, m)])
    key = np.unique((np.minimum(u, v) * V + np.maximum(u, v))[u != v])
    u, v = key // V, key % V
    w = rng.integers(1, 51, len(u)).astype(np.int32)
    key = np.concatenate([u * V + v, v * V + u])
    at = np.argsort(key, kind="stable")
    beg = np.concatenate([[0], np.cumsum(np.bincount(key // V, minlength=V))]).astype(np.int64)
    return G.Graph(beg, (key[at] % V).astype(np.int32), np.concatenate([w, w])[at])


@pytest.mark.parametrize("V,m,columns,hops", [
    (2_000_001, 1_200_000, 24, [None, 1, 2, 3, 4, 5, 6, 7, 8]),   # 1 mask word
    (2_000_002, 1_200_000, 84, [None, 3, 4]),                     # 3
    (2_000_003, 1_200_000, 136, [None, 2, 5]),                    # 5
    (2_000_003, 1_200_000, 240, [None, 4, 8]),                    # 8
    (2_000_001, 8_500_000, 240, [None]),                          # 8, two edge classes
])
def test_queries_keep_their_cost(V, m, columns, hops):
    g = _graph(V, m, V + columns)
    rng = np.random.default_rng(columns)
    grp = G.Groups.from_lists([rng.choice(V, int(rng.integers(1, 3000)), replace=False).tolist() for _ in range(columns)])
    qs = rng.permutation(columns).astype(np.int32).reshape(-1, 4)  # every group once
    got = []
    for search in (1, 0):
        eng = G.Engine(0, max_batch=16, batch_search=search)
        try:
            dg = eng.graph(g, grp)
            got.append([[(a.status, a.cost) for a in dg.solve_batch(list(qs), [h] * len(qs))] for h in hops])
            dg.close()
        finally:
            eng.close()
    for h, a, b in zip(hops, *got):
        assert a == b, h
    assert any(s == G.OK for a in got[0] for s, _ in a)


@pytest.mark.parametrize("D", [6, 7])
@pytest.mark.parametrize("V,m,smax,wmax", [(60, 150, 20, 5), (900, 4000, 4, 100), (2500, 5000, 60, 1 << 16)])
def test_pulled_rounds_of_the_other_bounds(engine, D, V, m, smax, wmax):
    g = G.synth_rmat(V, m, 7 + V, wmax=wmax)
    grp = G.synth_groups_uniform(g.V, 40, 1, smax, 8)
    rng = np.random.default_rng(9 + D)
    qs = [rng.choice(40, size=int(k), replace=False).astype(np.int32) for k in (1, 2, 3, 4, 5, 5, 6)]
    dg = engine.graph(g, grp)
    try:
        for q, a in zip(qs, dg.solve_batch(qs, [D] * len(qs))):
            assert (a.cost if a.ok else -1) == O.gst_hop(g, grp, q, D)["cost"], (q, D)
            if a.ok:
                assert G.verify_tree(g, grp, q, D, a.cost, a.edges, a.root) == 0
    finally:
        dg.close()
