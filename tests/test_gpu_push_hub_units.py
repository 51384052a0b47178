"""A round whose hub vertices do not fit the buffers that split them: more slots than
2^20 and more units (1024 neighbours each) than 2^22, the last of which would begin in
the buffer and end past it. What does not fit is pushed in place.

16,384 sources (256 chunks) point at one vertex, that one at 8,192 hubs, and every hub at
the same 2,049 vertices: the third round has 2.1 million hub items of three units each.
Its result is known: each hub keeps alpha (1 - alpha)^2 / 8192 of a source, each of the
last vertices holds (1 - alpha)^3 / 2049, a sum of 8,192 equal terms, each rounded by 2^-25
of it at most, always in the same direction at worst: 8192 2^-25 = 2.4e-4 of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SOURCES, HUBS, LEAVES, ALPHA = 16_384, 8_192, 2_049, 0.2


def test_hubs_past_the_buffers():
    import tsvd_gb300 as T
    relay = SOURCES
    hubs = relay + 1 + np.arange(HUBS)
    leaves = relay + 1 + HUBS + np.arange(LEAVES)
    n = int(leaves[-1]) + 1
    src = np.arange(SOURCES, dtype=np.int32)
    edges = np.concatenate([
        np.stack([src, np.full(SOURCES, relay)], 1),
        np.stack([np.full(HUBS, relay), hubs], 1),
        np.stack([np.repeat(hubs, LEAVES), np.tile(leaves, HUBS)], 1)]).astype(np.int32)
    with T.Session(n, src, directed=True, alpha=ALPHA, rmax=1e-9, n_parts=2, rank_d=2) as s:
        s.graph_insert(edges)
        for _ in range(2):  # the second time over buffers that the first has left
            s.ppr_refresh(1)
            s.ppr_push()
            rows = np.r_[0:3, 63:66, SOURCES // 2:SOURCES // 2 + 2, SOURCES - 3:SOURCES]
            p, r = s.ppr_state_rows(rows, which=1), s.ppr_state_rows(rows, which=0)
            want = ALPHA * (1 - ALPHA) ** 2 / HUBS
            assert np.abs(p[:, hubs] / want - 1).max() <= 1e-6
            want = (1 - ALPHA) ** 3 / LEAVES
            assert np.abs(r[:, leaves] / want - 1).max() <= 2.4e-4
            r[:, leaves] = 0
            assert not r.any()
