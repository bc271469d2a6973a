"""Trees whose groups lie 2^31 and more apart (heaviest weights along a path): the shared search
compares distances as signed words and knows of the farther ones only that they are farther, so
its queries prune with that and find the tree of a query that searches on its own.  Past
2^31 - 1 a cost no longer fits the result's word; both wrap alike."""
import numpy as np
import pytest

import gst_b200 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [100, 128, 129, 130, 180, 250])
@pytest.mark.parametrize("groups", [[[0], [-1]], [[0], [-1], [5]], [[0, 1], [-1, -2], [60], [90, 91]]])
def test_far_groups_keep_their_tree(V, groups):
    beg = np.concatenate([[0, 1], 1 + 2 * np.arange(1, V - 1), [2 * V - 2]]).astype(np.int64)
    adj = np.concatenate([[1], np.stack([np.arange(V - 2), np.arange(2, V)], 1).ravel(), [V - 2]]).astype(np.int32)
    g = G.Graph(beg, adj, np.full(2 * V - 2, 1 << 24, np.int32))
    grp = G.Groups.from_lists([[v % V for v in s] for s in groups])
    q = np.arange(len(groups), dtype=np.int32)
    got = []
    for search in (1, 0):
        eng = G.Engine(0, batch_search=search)
        dg = eng.graph(g, grp)
        got += [dg.solve(q), dg.solve_batch([q], [None])[0]]
        dg.close()
        eng.close()
    want = got[2]
    lo, hi = max(groups[0]), V + min(groups[1])
    assert want.ok and want.edges.tolist() == [[v, v + 1, 1 << 24] for v in range(lo, hi)]
    for a in got:
        assert (a.status, a.cost, a.edges.tolist()) == (want.status, want.cost, want.edges.tolist())
