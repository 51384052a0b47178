"""Pair scores (lp_score_kernel) at ranks that are and are not multiples of four,
for one pair to more than the grid has groups of lanes. Sums of d doubles: 1e-12 of
the largest score; a faulty pair anywhere is an error, and the next call is fine."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 5, 32, 50, 100])
def test_pair_scores(d):
    import tsvd_gb300 as T
    n = 3001
    edges = T.rmat_edges(n, 24000, seed=2)
    src = T.sample_sources(n, edges, 120, seed=2)
    with T.Session(n, src, directed=True, alpha=0.2, rmax=1e-5, n_parts=4, rank_d=d,
                   transform=T.TRANSFORM_LOG10_LP, root_scaling=T.ROOT_U, lp_right_factor=True,
                   dirty_rule=T.DIRTY_ALL) as s:
        s.step(edges)
        U, V = s.embedding(), s.lp_right_factor().astype(np.float64)
        deg_i, deg_j = s.degrees(0)[0], s.degrees(1)[0]
        row = {int(v): i for i, v in enumerate(src)}
        rng = np.random.default_rng(d)
        for m in (1, 3, 31, 4000, 60000):
            pairs = np.stack([rng.choice(src, m), rng.integers(0, n, m)], 1).astype(np.int32)
            ref = np.einsum("kd,kd->k", U[[row[int(i)] for i in pairs[:, 0]]], V[pairs[:, 1]])
            for scaled in (False, True):
                if scaled:
                    ref = ref * deg_i[pairs[:, 0]] * deg_j[pairs[:, 1]]
                got = s.lp_scores(pairs, degree_scaled=scaled)
                assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max() + 1e-300
            bad = pairs.copy()
            bad[m // 2, 1] = n
            with pytest.raises(T.TsvdError):
                s.lp_scores(bad)
