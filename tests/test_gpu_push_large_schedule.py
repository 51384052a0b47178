"""The push of a large graph (its rounds launched as a graph, whose parameters change with
the threshold level and with the adjacency) with the hub threshold schedule, and with one
for every vertex, through three snapshots: 350,005 (vertex, chunk) pairs, hubs of
thousands of neighbours. The check, with its tolerance, is that of the other layouts."""
import pytest

from test_gpu_push_layout import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("schedule", [
    dict(push_levels=3, push_ratio=4.0, push_hub_degree=200),
    dict(push_levels=2, push_ratio=8.0)])
def test_schedule_on_a_large_graph(schedule, directed):
    import tsvd_gb300 as T
    n, rmax = 70_001, 1e-6
    edges = T.rmat_edges(n, 500_000, directed=directed, seed=7)
    cut = [0, len(edges) * 6 // 10, len(edges) * 8 // 10, len(edges)]
    src = T.sample_sources(n, edges[:cut[1]], 300, seed=7)
    with T.Session(n, src, directed=directed, alpha=0.2, rmax=rmax, n_parts=2, rank_d=4,
                   dynamic_ppr_start_iter=2, **schedule) as s:
        for it in range(1, 4):
            s.graph_insert(edges[cut[it - 1]:cut[it]])
            for t in range(2 if directed else 1):
                s.ppr_refresh(it, bool(t))
                s.ppr_push(bool(t))
        _check(T, s, n, directed, 0.2, rmax)
