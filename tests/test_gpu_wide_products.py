"""The products of merges wider than 256 columns (csrc/sgemm.cu) at the edges of
their 128 x 64 tiles and 16-value slices: rows and columns that are or are not
multiples of four, K split over CTAs or not, fewer rows than columns.

The matrix has rank 40, which the subspace iteration finds at once. B B^T is twice
off by: the basis V, 256 2^-24 = 1.5e-5; the products, sqrt(2048) 2^-24 = 2.7e-6;
the eigenvectors' length, 4.4e-5 (jacobi.cu). Together 1.3e-4.

A single matrix with many more columns than rows is refused, as its basis has more
rows than the Gram's scratch is made for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [
    (41, 257), (63, 300), (128, 260), (129, 303), (255, 512), (256, 513), (257, 400),
    (1500, 1024), (1501, 1030), (1499, 2048), (4000, 259)])
def test_wide_merge_of_a_low_rank_matrix(rows, cols):
    import tsvd_gb300 as T
    rng = np.random.default_rng(cols)
    u = np.linalg.qr(rng.standard_normal((rows, 40)))[0] * np.geomspace(100, 1, 40)
    M = (u @ np.linalg.qr(rng.standard_normal((cols, 40)))[0].T).astype(np.float32)
    M = M.astype(np.float64)
    if cols > 128 * (-(-rows // 128) + 1) and rows >= 255:
        with pytest.raises(T.TsvdError, match="gram: work buffer too small"):
            T.merge_svd(M, 40)
        return
    US, sig = T.merge_svd(M, 40)
    u0, s0, _ = np.linalg.svd(M, full_matrices=False)
    E = u0[:, :40] * s0[:40]
    r = np.linalg.qr(np.concatenate([US, E], axis=1))[1]
    rb, re = r[:, :40], r[:, 40:]
    assert np.linalg.norm(rb @ rb.T - re @ re.T) <= 1.3e-4 * np.linalg.norm(re @ re.T)
    assert np.abs(sig / s0[:40] - 1).max() <= 1.3e-4
