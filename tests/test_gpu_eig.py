"""The one-sided Jacobi eigen-solver (csrc/eig.cu) behind the tree merges, at
the sizes where its layout changes: one column per block, odd and even block
widths, the padding of the panel factorization (multiples of 32 and one past),
1-8 CTAs per problem, 8 and 16 lanes per column pair, the largest size; and
merges with fewer rows than columns, whose Grams are singular.

Every inner node of the tree is checked against the exact truncated SVD of its
children's factors. Tolerance: a column takes part in at most about 255
rotations a sweep and 8 sweeps, each rounding it by 2^-24 at random, so its
direction and length are off by sqrt(2040) 2^-24 = 2.7e-6; four times that."""
import numpy as np
import pytest

from oracle.tree_oracle import frpca as oracle_frpca, gaussian_matrix

pytestmark = pytest.mark.gpu
TOL = 1.1e-5


@pytest.mark.parametrize("d,h,sources", [
    (1, 2, 300), (9, 2, 300), (16, 2, 300), (17, 2, 300), (33, 2, 300), (80, 2, 300),
    (81, 2, 300), (85, 3, 300), (96, 2, 300), (128, 2, 300), (64, 4, 300), (32, 2, 40)])
def test_merges_match_exact_svd(d, h, sources):
    import tsvd_gb300 as T
    n, parts = 3000, h * h
    edges = T.rmat_edges(n, 24000, seed=5)
    src = T.sample_sources(n, edges, sources, seed=5)
    with T.Session(n, src, n_parts=parts, hierarchy_n=h, rank_d=d, alpha=0.2, rmax=1e-5,
                   transform=T.TRANSFORM_LN_N, passes_q=4) as s:
        s.step(edges)
        for node in range(1, 1 + h):
            M = np.concatenate([s.tree_factor(node * h + 1 + c)[0] for c in range(h)], axis=1)
            B, sig = s.tree_factor(node)
            u, s0, _ = np.linalg.svd(M, full_matrices=False)
            us = u[:, :d] * s0[:d]
            exact = us @ us.T
            assert np.isfinite(B).all()
            err = np.linalg.norm(B @ B.T - exact) / np.linalg.norm(exact)
            assert err <= TOL, (node, err)
            big = s0[:d] > 1e-5 * s0[0]
            assert np.abs(sig[big] / s0[:d][big] - 1).max() <= TOL, node


def test_blocks_of_low_rank_stay_finite():
    """Blocks with fewer non-empty columns, or sources, than the basis is wide:
    their Grams are singular, and most columns of the factor are dropped."""
    import tsvd_gb300 as T
    n, parts, d = 20000, 64, 128
    edges = T.rmat_edges(n, 60000, seed=9)
    src = T.sample_sources(n, edges, 150, seed=9)
    with T.Session(n, src, n_parts=parts, rank_d=d, alpha=0.2, rmax=1e-4) as s:
        s.step(edges)
        info = s.block_info()
        assert info["nnz"].min() < 133 * 150  # some blocks cannot fill the basis
        for node in range(2 * parts - 1):
            B, sig = s.tree_factor(node)
            assert np.isfinite(B).all() and np.isfinite(sig).all(), node
            assert (np.diff(sig) <= 1e-6 * sig[0]).all(), node


@pytest.mark.parametrize("k", [1, 26, 27, 28, 59, 60, 91, 92, 123, 124, 128, 139])
def test_frpca_basis_at_the_panel_edges(k):
    """CholeskyQR's factor and inverse (csrc/chol.cu) at basis widths k + 5
    around its 32-column panels: U = Q V is orthonormal. Two passes leave Q
    orthonormal to about l 2^-24 = 9e-6, V's columns are up to 4.4e-5 short;
    their sum, doubled for the squares, is 1.1e-4."""
    import tsvd_gb300 as T
    rng = np.random.default_rng(k)
    m, n = 300, 500
    q1 = np.linalg.qr(rng.standard_normal((m, m)))[0]
    q2 = np.linalg.qr(rng.standard_normal((n, m)))[0]
    A = (q1 * np.geomspace(10, 0.1, m)) @ q2.T
    U, S, V = T.frpca(np.arange(m + 1) * n, np.tile(np.arange(n), m), A.ravel(), (m, n), k, 6)
    assert np.abs(U.T @ U - np.eye(k)).max() <= 1.1e-4
    # frPCA's own values, not the matrix's: a few passes over a slow decay
    S0 = oracle_frpca(A, k, 6, omega=gaussian_matrix(20231, 0, n, k + 5))[1][::-1]
    lead = max(1, k // 2)
    assert np.allclose(S[:lead], S0[:lead], rtol=2e-3)
