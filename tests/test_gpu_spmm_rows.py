"""The FP32 sparse products (csrc/plain.cu) at the lengths and counts of rows
where their split changes: remainders of the eight entries in flight, rows that a
warp or all warps of a CTA take, one to eight rows a CTA, the three widths of a
subgroup of lanes, empty rows.

The columns are multiples of eight vectors, so frPCA with k >= 8 gives the matrix
back: up to the vectors' length (4.4e-5 each, see jacobi.cu) times its norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SUPPORT = (1, 2, 7, 9, 65, 131, 513, 700)


@pytest.mark.parametrize("cols", [17, 640, 5003])
@pytest.mark.parametrize("k", [8, 60, 100, 128])
def test_products_give_a_low_rank_matrix_back(cols, k):
    import tsvd_gb300 as T
    rng = np.random.default_rng(cols)
    m = 720
    base = np.zeros((m, 8))
    for j, n in enumerate(SUPPORT):
        base[rng.choice(700, n, replace=False), j] = rng.choice([-1.0, 1.0], n) / np.sqrt(n)
    A = base[:, np.arange(cols) % 8] * rng.uniform(0.5, 1.5, cols)
    A = A.astype(np.float32).astype(np.float64)
    r, c = np.nonzero(A)
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=m))])
    for q in (3, 4):
        U, S, V = T.frpca(rp, c, A[r, c], A.shape, k, q, fp32=True)
        assert np.abs(U * S @ V.T - A).max() <= 2 * 4.4e-5 * np.linalg.norm(A, 2)
