"""Starting queries together (k_admit) and the sizes of their row pools: a tight memory budget
(a pool of an eighth of the vertices that the heavy queries overflow, then the dense layout),
a wide one (a mapped pool of up to one row per vertex), and batches whose queries start from a
shared search, from cached groups, from both and alone, all give the reference's costs."""
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
