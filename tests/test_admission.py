"""Starting queries together (k_admit) and the sizes of their row pools: a tight memory budget
(a pool of an eighth of the vertices that the heavy queries overflow, then the dense layout),
a wide one (a mapped pool of up to one row per vertex), and batches whose queries start from a
shared search, from cached groups, from both and alone, all give the reference's costs.
Queries beyond one search's 64 wait for the next search; without memory for a search's table
they search on their own."""
import numpy as np
import pytest

import gst_b200 as G
from conftest import golden_inputs, load_golden
from test_gpu_parity import _check, _ref, consensus

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget", [3 << 30, 0])
@pytest.mark.parametrize("slots", [1, 5])
def test_pool_sizes_keep_the_optima(budget, slots):
    fx = load_golden("c2_rmat170k_k5k7")
    g, grp = golden_inputs(fx)
    eng = G.Engine(0, mem_budget_bytes=budget, max_batch=slots)
    try:
        dg = eng.graph(g, grp)
        todo = [(q, c["hop"], w) for c in fx["cases"] for q, w in list(zip(c["queries"], consensus(c)))[:6] if w]
        for (q, h, w), a in zip(todo, dg.solve_batch([x[0] for x in todo], [x[1] for x in todo])):
            _check(g, grp, q, h, a, _ref(w))
        dg.close()
    finally:
        eng.close()


@pytest.mark.parametrize("search", [0, 1])
def test_mixed_starts_keep_the_optima(search):
    fx = load_golden("rmat50k_hop")
    g, grp = golden_inputs(fx)
    eng = G.Engine(0, max_batch=16, batch_search=search)
    try:
        dg = eng.graph(g, grp)
        cases = [c for c in fx["cases"] if c["hop"] in (2, 4)]
        todo = [(q, c["hop"], w) for c in cases for q, w in list(zip(c["queries"], consensus(c)))[:8] if w]
        some = sorted({int(i) for q, h, _ in todo[::2] for i in q if h == 4})  # all or some of a query's
        dg.cache_warm_hop(some, 4, 1 << 30)
        for (q, h, w), a in zip(todo, dg.solve_batch([x[0] for x in todo], [x[1] for x in todo])):
            _check(g, grp, q, h, a, _ref(w))
        for q, h, w in todo[:4]:
            _check(g, grp, q, h, dg.solve(q, h), _ref(w))
        dg.close()
    finally:
        eng.close()


@pytest.mark.parametrize("budget", [0, 60 << 20])
@pytest.mark.parametrize("slots", [1, 7, 32])
def test_more_queries_than_one_search(budget, slots):
    g = G.synth_rmat(30_000, 120_000, 41)
    grp = G.synth_groups_zipf(g.V, 500, 1.5, 1, 40, 42)
    rng = np.random.default_rng(43)
    qs = [rng.choice(500, size=int(rng.integers(2, 5)), replace=False).astype(np.int32) for _ in range(90)]
    hops = [None if x < 0.5 else int(rng.integers(0, 4)) for x in rng.random(90)]
    ref = G.Engine(0, batch_search=0)
    eng = G.Engine(0, max_batch=slots, mem_budget_bytes=budget)
    try:
        alone = ref.graph(g, grp)
        dg = eng.graph(g, grp)
        want = [(a.status, a.cost) for a in (alone.solve(q, h) for q, h in zip(qs, hops))]
        got = dg.solve_batch(qs, hops)
        assert [(a.status, a.cost) for a in got] == want
        if budget == 0:
            sv = dg.server()
            tickets = [sv.submit(q, h) for q, h in zip(qs, hops)]
            assert [(a.status, a.cost) for a in map(sv.wait, tickets)] == want
            sv.close()
        alone.close()
        dg.close()
    finally:
        ref.close()
        eng.close()
