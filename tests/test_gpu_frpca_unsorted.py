"""tsvd_frpca_fp32 over matrices whose rows do not ascend, hold zeros or hold an entry
twice: they are sorted and stripped on the device, by column and then by row, and every
sum is in a fixed order, so the results have the bits that the same entries in order
give. Sizes at the byte edges of the radix sort: the number of passes decides which of
the two buffers holds the result; rows and columns that are empty, at either end too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [
    (1, 300), (40, 254), (255, 255), (256, 256), (257, 257), (300, 66_000), (66_000, 300)])
@pytest.mark.parametrize("mixed,zeros", [(True, False), (False, True), (True, True)])
def test_same_bits_as_in_order(rows, cols, mixed, zeros):
    import tsvd_gb300 as T
    rng = np.random.default_rng(rows + cols)
    n = 40 * max(rows, cols) // 8
    r = np.sort(rng.integers(0, rows, n))
    r = r[(r % 7 != 0) | (rows == 1)]  # empty rows, the first one among them
    c = rng.integers(1, max(2, cols - 1), len(r))  # and columns; some entries twice
    v = rng.standard_normal(len(r))
    v0 = np.where(rng.random(len(r)) < 0.1, np.where(rng.random(len(r)) < 0.5, 0.0, -0.0), v)
    v = v0 if zeros else v
    order = np.lexsort((np.arange(len(r)), c, r))  # entries given twice keep their order
    keep = order[v[order] != 0]
    given = np.arange(len(r)) if mixed else order

    def csr(at):
        return np.concatenate([[0], np.cumsum(np.bincount(r[at], minlength=rows))]), c[at], v[at]

    k = min(8, rows)
    want = T.frpca(*csr(keep), (rows, cols), k, 4, fp32=True)
    got = T.frpca(*csr(given), (rows, cols), k, 4, fp32=True)
    assert np.isfinite(want[1]).all() and want[1][0] > 0
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
