"""tsvd_frpca and tsvd_frpca_fp32 over every form of one matrix: rows in or out of
order, explicit zeros, 0- and 1-based, entries before the first row, empty rows
and columns, one entry; sparse rows that do not ascend, or that hold zeros, are
built on the host, the others on the device, with the same values in the same
order. And the errors of a walk over the entries, in the order of the walk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
M, N, RANK = 60, 700, 30


def _matrix():
    """Half of the rows and some columns (the first and the last) empty."""
    rng = np.random.default_rng(3)
    A = np.where(rng.random((M, N)) < 0.2, rng.standard_normal((M, N)) * 3, 0.0)
    A[1::2] = 0
    A[:, [0, 5, 6, 7, 300, N - 1]] = 0
    return A


def _csr(A, order="sorted", zeros=False, base=0, lead=0):
    rng = np.random.default_rng(7)
    rp, ci, va = [0], [], []
    for row in A:
        c = np.flatnonzero(row)
        if zeros:
            c = np.union1d(c, rng.choice(len(row), 9))
        if order == "mixed":
            c = rng.permutation(c)
        ci.append(c)
        va.append(row[c])
        rp.append(rp[-1] + len(c))
    ci = np.concatenate([np.full(lead, 10 ** 6)] + ci).astype(np.int32)
    va = np.concatenate([np.full(lead, np.nan)] + va)
    return np.array(rp) + lead + base, ci + base, va


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("order,zeros,base,lead", [
    ("sorted", False, 0, 0), ("sorted", False, 1, 5), ("mixed", False, 0, 3),
    ("sorted", True, 1, 0), ("mixed", True, 0, 0)])
def test_every_form_of_a_matrix(order, zeros, base, lead, fp32):
    import tsvd_gb300 as T
    A = _matrix()
    rp, ci, va = _csr(A, order, zeros, base, lead)
    U, S, V = T.frpca(rp, ci, va, A.shape, RANK, 4, index_base=base, fp32=fp32)
    # k is the matrix's rank: the product is the matrix, up to the inputs' rounding
    # (2^-11 of an entry in halves) and the vectors' length (4.4e-5, see jacobi.cu)
    tol = (0 if fp32 else 2.0 ** -11) * np.abs(A).max() + 2 * 4.4e-5 * np.linalg.norm(A, 2)
    assert np.abs(U * S @ V.T - A).max() <= tol
    assert not V[[0, 5, 6, 7, 300, N - 1]].any()
    if fp32:  # SpMM and every other sum in a fixed order: the same bits
        U0, S0, V0 = T.frpca(*_csr(A), A.shape, RANK, 4, fp32=True)
        assert np.array_equal(U, U0) and np.array_equal(S, S0) and np.array_equal(V, V0)


@pytest.mark.parametrize("fp32", [False, True])
def test_smallest_matrices(fp32):
    import tsvd_gb300 as T
    U, S, V = T.frpca([0, 0], [], [], (1, 1), 1, 1, fp32=fp32)
    assert not U.any() and not S.any() and not V.any()
    U, S, V = T.frpca([0, 1, 2], [4, 4], [0.0, 0.0], (2, 9), 2, 1, fp32=fp32)
    assert not U.any() and not S.any() and not V.any()
    U, S, V = T.frpca([0, 0, 1], [4], [-3.0], (2, 9), 1, 2, fp32=fp32)
    assert abs(S[0] - 3) <= 1e-5 and abs((U * S @ V.T)[1, 4] + 3) <= 1e-5


@pytest.mark.parametrize("fp32", [False, True])
def test_the_first_fault_is_named(fp32):
    import tsvd_gb300 as T
    A = _matrix()
    for faults, message in [({"col": 9}, "column out of range"), ({"nan": 9}, "non-finite"),
                            ({"big": 9}, "float range"), ({"nan": 4, "col": 9}, "non-finite"),
                            ({"nan": 9, "col": 4}, "column out of range"),
                            ({"rp": 2, "nan": 4}, "non-finite"), ({"rp": 2}, "row pointers")]:
        rp, ci, va = _csr(A)
        for what, at in faults.items():
            if what == "col":
                ci[at] = N
            elif what == "rp":
                rp[at + 1] = rp[at] - 1
            else:
                va[at] = np.nan if what == "nan" else 1e39
        with pytest.raises(Exception, match=message):
            T.frpca(rp, ci, va, A.shape, 4, 2, fp32=fp32)
    with pytest.raises(Exception, match="k=0"):
        T.frpca(*_csr(A), A.shape, 0, 2, fp32=fp32)
