"""What a round of the push reads late has received what was scattered early: a vertex
of up to 1024 neighbours scatters at once, and it keeps its place among the items.
Which of the many valid states a push ends in hangs on it, and the push identity, which
holds in all of them, does not see it; the number of pushes does.

One source points at `items` vertices, so the second round pushes them all. Some of them
are parents of `degree` others each, every other one has one parent and points at a
vertex of its own without out-neighbours. A child is pushed again in the third round
unless it was read after its parent had scattered. The items come in no particular
order and the grid takes them in k = items / (warps of 8 blocks an SM) passes, so of the
children about (1 - 1/k) / 2 are a pass or more behind their parent: 0.33 of them at
30,000 items, 0.46 at 120,000. Some passes go by while a parent scatters (1024
neighbours take a warp 30 us, two or three passes of such items), so a third of that is
asked for: 0.1. If the parents waited for the end of the round, no child would have seen
its parent; if they came last in it, 0.02 of them at most."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("items,degree", [
    (30_000, 129),   # 60,001 pairs: a small graph
    (60_000, 300),   # 120,001 pairs: a large one
    (120_000, 1024),  # the longest list that is scattered at once
])
def test_late_items_see_early_scatters(items, degree):
    import tsvd_gb300 as T
    rng = np.random.default_rng(degree)
    n = 2 * items + 1
    child = rng.permutation(np.arange(1, items + 1))
    parents = items // (degree + 1)
    groups = child[:parents * (degree + 1)].reshape(parents, degree + 1)
    leaves = np.setdiff1d(child, groups[:, 0])
    edges = np.concatenate([
        np.stack([np.zeros(items, int), np.arange(1, items + 1)], 1),
        np.stack([np.repeat(groups[:, 0], degree), groups[:, 1:].ravel()], 1),
        np.stack([leaves, leaves + items], 1)]).astype(np.int32)
    src = np.concatenate([[0], items + 1 + np.arange(7)]).astype(np.int32)
    with T.Session(n, src, directed=True, alpha=0.2, rmax=1e-9, n_parts=2, rank_d=2) as s:
        s.graph_insert(edges)
        s.ppr_refresh(1)
        s.ppr_push()
        again = s.stats()["pushes"] - 1 - items
    waited = again / (parents * degree)
    assert waited <= 1
    assert 1 - waited >= 0.1, waited
