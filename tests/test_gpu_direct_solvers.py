"""What the direct entry points' eigen-solvers are each taken for.

Up to 256 columns, the two-sided solver (csrc/jacobi.cu): left singular vectors M V / s
of a matrix whose columns have very different norms. It leaves a pair alone below 1e-11
of the largest eigenvalue, so vectors i and j may have 1e-11 s_1^2 / (s_i s_j) of each
other, and its rotations shorten a vector by 4.4e-5 n / 256 at n columns, twice that in
a product of two. A solver whose V is good to 2^-24 of a column, and not of each entry,
leaves 2^-24 s_1 / s_k of the first vector in the k-th: 6e-5 at 1e-3.

Wider, the one-sided solver (csrc/eig.cu) after the subspace iteration, with columns of
the basis beyond the matrix's rank: each singular value to 1.1e-5, its tolerance in
test_gpu_eig.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(300, 16), (300, 32), (1000, 48), (1000, 49)])
def test_left_vectors_of_a_graded_matrix(rows, cols):
    import tsvd_gb300 as T
    rng = np.random.default_rng(rows + cols)
    M = rng.standard_normal((rows, cols)) * np.geomspace(1e3, 1e-3, cols)
    M = M.astype(np.float32).astype(np.float64)
    US, sig = T.merge_svd(M, cols)
    s0 = np.linalg.svd(M, compute_uv=False)
    big = s0 > 1e-4 * s0[0]
    x = s0[big] / s0[0]
    U = US[:, big] / s0[big]
    tol = 2 * 4.4e-5 * cols / 256 + 1e-11 / np.outer(x, x)
    assert (np.abs(U.T @ U - np.eye(len(x))) <= tol).all()


@pytest.mark.parametrize("rows,cols,rank", [(600, 400, 133), (1500, 512, 170)])
def test_wide_merge_below_full_rank(rows, cols, rank):
    import tsvd_gb300 as T
    rng = np.random.default_rng(rows + cols)
    u = np.linalg.qr(rng.standard_normal((rows, rank)))[0] * np.geomspace(10, 1, rank)
    M = (u @ np.linalg.qr(rng.standard_normal((cols, rank)))[0].T).astype(np.float32)
    M = M.astype(np.float64)
    US, sig = T.merge_svd(M, 64)
    s0 = np.linalg.svd(M, compute_uv=False)[:64]
    assert np.abs(sig / s0 - 1).max() <= 1.1e-5
