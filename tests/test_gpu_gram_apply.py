"""The Gram and X W kernels (csrc/dense.cu) behind tsvd_merge_svd and tsvd_frpca
at the edges of their tiles: rows around the 32 of a staged slab, the 128 of a
row chunk and the count from which 128-row tiles fill the SMs; columns around
the 4 x 4 output tiles and the 32-deep slabs; columns of very different norms,
and norms whose squares are near the end of the float range.

Tolerance of the products of factors: the eigen-solver's 1.1e-5 (about 2040
rotations of 2^-24 each, as a random walk, four times over), to which X W adds
sqrt(48) 2^-24 = 4e-7. Bases: two passes of CholeskyQR leave l 2^-24 = 1.5e-6
and V's rotations 2.7e-6; ten times their sum, as several kernels follow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1.2e-5


@pytest.mark.parametrize("rows,cols,scale", [
    (5, 5, 1.0), (31, 3, 1.0), (32, 4, 1.0), (33, 5, 1.0), (127, 31, 1.0), (128, 32, 1.0),
    (129, 33, 1.0), (300, 48, 1.0), (19329, 7, 1.0), (19457, 48, 1.0), (300, 9, 2.0 ** 62),
    (300, 9, 2.0 ** -40)])
def test_merge_of_one_matrix(rows, cols, scale):
    import tsvd_gb300 as T
    rng = np.random.default_rng(rows + cols)
    M = rng.standard_normal((rows, cols))
    M *= 3 * np.geomspace(1, 1e-3, cols) / np.linalg.norm(M, axis=0)
    M = (M * scale).astype(np.float32).astype(np.float64)
    d = min(rows, cols)
    US, sig = T.merge_svd(M, d)
    u, s0, _ = np.linalg.svd(M / scale, full_matrices=False)
    B = US / scale
    # |B B^T - E E^T| over |E E^T| through the small cores of [B E]
    E = u * s0
    q, r = np.linalg.qr(np.concatenate([B, E], axis=1))
    rb, re = r[:, :d], r[:, d:]
    err = np.linalg.norm(rb @ rb.T - re @ re.T) / np.linalg.norm(re @ re.T)
    assert np.isfinite(US).all()
    assert err <= TOL, err
    big = s0 > 1e-5 * s0[0]
    assert np.abs(sig[big] / scale / s0[big] - 1).max() <= TOL


@pytest.mark.parametrize("cols", [1009, 20011])
def test_frpca_bases_over_many_columns(cols):
    import tsvd_gb300 as T
    rng = np.random.default_rng(cols)
    m, k = 64, 20
    q1 = np.linalg.qr(rng.standard_normal((m, m)))[0]
    q2 = np.linalg.qr(rng.standard_normal((cols, m)))[0]
    A = (q1 * np.geomspace(10, 0.1, m)) @ q2.T
    U, S, V = T.frpca(np.arange(m + 1) * cols, np.tile(np.arange(cols), m), A.ravel(), (m, cols),
                      k, 6)
    assert np.abs(U.T @ U - np.eye(k)).max() <= 4.2e-5
    assert np.abs(V.T @ V - np.eye(k)).max() <= 4.2e-5
