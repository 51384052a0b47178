"""tsvd_frpca_fp32 where the device has room for the matrix (16 bytes an entry) and the
call's work, but not for what building the matrix there takes (44) beside that work: the
matrix is then built on the host, with the same bits.

4 million entries: 64 MB, built on the device 180 MB; work for 20,000 columns some 124
MB. 245 MB are left free, halfway between 188 and 304."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_sparse_form_on_a_nearly_full_device():
    import torch
    import tsvd_gb300 as T
    rows, cols, per_row, k = 600, 20_000, 6_667, 32
    rng = np.random.default_rng(1)
    ci = np.concatenate([np.sort(rng.choice(cols, per_row, replace=False)) for _ in range(rows)])
    a = (np.arange(rows + 1) * per_row, ci, rng.standard_normal(rows * per_row), (rows, cols), k, 4)
    want = T.frpca(*a, fp32=True)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - 245 * 2 ** 20, dtype=torch.uint8, device="cuda")
    try:
        got = T.frpca(*a, fp32=True)
    finally:
        del hold
        torch.cuda.empty_cache()
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
