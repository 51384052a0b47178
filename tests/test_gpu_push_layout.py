"""The push at the sizes where its work is laid out differently: a bitset of a
few words and a graph smaller than a warp's 256 pairs (collect_kernel's words
per warp, pairs of several chunks in one word), hubs on both sides of the
light-item degree and of the small-round piece (128) in a chain of grown
snapshots (the launch graph's parameters change), and rounds of more than 2^18
items (pieces of 1024). Checked by the push identity, which holds in any push
order, and by the threshold.

The identity's tolerance is the 2e-5 of the other push tests, or, where it is
more, what fp32 residues can lose: a cell takes at most one addition a round
from each of its d neighbours, each rounded by 2^-25 of the residue there, and
the residues pushed to it add up to (1 - alpha) / alpha over the rounds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(T, s, n, directed, alpha, rmax):
    from helpers import push_identity_residual, transition
    for t in range(2 if directed else 1):
        off, nb = s.adjacency(t)
        P, deg = transition(n, off, nb)
        p, r = s.ppr_state(bool(t), 1), s.ppr_state(bool(t), 0)
        tol = max(2e-5, 2.0 ** -25 * deg.max() * (1 - alpha) / alpha) if n > 10_000 else 2e-5
        assert push_identity_residual(p, r, s.sources, P, alpha) < tol
        assert (r[:, deg > 0] <= np.float32(rmax)).all()
        assert (p >= 0).all()


@pytest.mark.parametrize("n,m,sources,rmax,schedule", [
    (33, 90, 20, 1e-6, {}),                # 3 words, one chunk
    (40, 200, 40, 1e-6, {}),
    (100, 900, 90, 1e-6, {}),              # two chunks, pairs of both in one word
    (3001, 40_000, 129, 1e-6, {}),         # 3 chunks; hubs of several hundred neighbours
    (3001, 40_000, 129, 1e-6, dict(push_levels=3, push_ratio=4.0, push_hub_degree=200)),
    (70_001, 500_000, 300, 1e-6, {}),      # 350,005 pairs: dense rounds pass 2^18 items
])
@pytest.mark.parametrize("directed", [False, True])
def test_push_layouts(n, m, sources, rmax, schedule, directed):
    import tsvd_gb300 as T
    edges = T.rmat_edges(n, m, directed=directed, seed=n)
    cut = [0, len(edges) * 6 // 10, len(edges) * 8 // 10, len(edges)]
    src = T.sample_sources(n, edges[:cut[1]], min(sources, n // 2), seed=n)
    with T.Session(n, src, directed=directed, alpha=0.2, rmax=rmax, n_parts=2, rank_d=4,
                   dynamic_ppr_start_iter=2, **schedule) as s:
        for it in range(1, 4):
            s.graph_insert(edges[cut[it - 1]:cut[it]])
            for t in range(2 if directed else 1):
                s.ppr_refresh(it, bool(t))
                s.ppr_push(bool(t))
            if n < 10_000 or it == 3:
                _check(T, s, n, directed, 0.2, rmax)
