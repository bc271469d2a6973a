"""The shared distance search in two edge classes (light edges to a fixpoint, then the heavy
ones from every vertex that changed since): its order restated on the CPU against exact
distances, and on the GPU the same costs as one query at a time, which searches in one class."""
import numpy as np
import pytest

import gst_b200 as G
from test_shared_search_model import INF, _bf


def two_class_search(g, sets, queries, light):
    """Distances and column cutoffs; stars at every announced vertex before each step."""
    C, tail, w = len(sets), np.repeat(np.arange(g.V), np.diff(g.beg_pos)), g.weight.astype(np.uint64)
    d = np.full((C, g.V), INF, dtype=np.uint64)
    now, later = np.zeros((C, g.V), bool), np.zeros((C, g.V), bool)
    for c, s in enumerate(sets):
        d[c, s], now[c, s] = 0, True
    cut = np.full(C, INF, dtype=np.uint64)
    while now.any() or later.any():
        heavy = not now.any()
        act, now = (later, now) if heavy else (now, np.zeros_like(now))
        later = np.zeros_like(later) if heavy else later | act
        at = act.any(axis=0)
        stars = [d[q][:, at].sum(axis=0).min() for q in queries]
        for c in range(C):
            mine = [s for q, s in zip(queries, stars) if c in q]
            cut[c] = min(cut[c], max(mine)) if mine else cut[c]
        src, nd = d.copy(), d.copy()
        for c in range(C):
            e = act[c][tail] & ((w > light) if heavy else (w <= light)) & (src[c][tail] + w <= cut[c])
            np.minimum.at(nd[c], g.adj[e], src[c][tail[e]] + w[e])
            now[c] |= (nd[c] < d[c]) & (nd[c] < cut[c])
        d = nd
    return d, cut


@pytest.mark.parametrize("light", [0, 1, 13, 100])
def test_two_classes_reach_the_exact_distances(light):
    for seed in range(3):
        g = G.synth_rmat(200, 700, 10 + seed)
        grp = G.synth_groups_uniform(g.V, 9, 1, 4, 20 + seed)
        sets = [grp.members[grp.grp_ptr[i]:grp.grp_ptr[i + 1]] for i in range(9)]
        d, cut = two_class_search(g, sets, [[0, 1, 2], [2, 3, 4, 5], [6, 7, 8]], light)
        exact = _bf(g.beg_pos, g.adj, g.weight, sets)
        for c in range(9):
            near = exact[c] <= cut[c]
            assert (d[c][near] == exact[c][near]).all() and (d[c][~near] > cut[c]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("wmax", [1, 7, 100, 1 << 22])
def test_batch_in_two_classes_equals_one_at_a_time(wmax):
    eng = G.Engine(0, max_batch=32)
    try:
        g = G.synth_rmat(150_000, 5_200_000, 31, wmax=wmax)  # 15 sectors x 10M edges: two classes
        grp = G.synth_groups_zipf(g.V, 4000, 1.5, 1, 300, 32)
        dg = eng.graph(g, grp)
        qs = [q for k in (3, 5, 6) for q in G.synth_queries(grp.n_groups, 9, k, 33 + k)]
        for q, a in zip(qs, dg.solve_batch(qs, [None] * len(qs))):
            b = dg.solve(q)
            assert a.ok and b.ok and a.cost == b.cost, q
            assert G.verify_tree(g, grp, q, -1, a.cost, a.edges, a.root) == 0
        dg.close()
    finally:
        eng.close()
