"""A^T y, A x and the residual of a Newton solve (k_row_sums) over rows of every length around
its segments of 32 entries and blocks of 32 rows, very long ones and empty ones among them. The
mixed mode solves with FP32 fronts and refines with that residual: a sum that missed or doubled
an entry could not come to 1e-11 of the right-hand side."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _matrix(m, n, lengths, seed):
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for i, len_i in enumerate(lengths):
        c = rng.choice(n, size=min(n, len_i), replace=False)
        rows += [i] * c.size
        cols += list(c)
    A = sp.csr_matrix((rng.standard_normal(len(rows)) / np.sqrt(1.0 + np.asarray(lengths)[rows]), (rows, cols)), (m, n))
    A = A.tolil()
    for i in range(min(m, n)):                 # a dominant entry, where a row has any
        if lengths[i]:
            A[i, (7 * i) % n] = 2.0
    A = A.tocsr()
    A.sort_indices()
    return A


LENGTHS = {
    "segments": [1, 31, 32, 33, 63, 64, 65, 96, 8, 7, 9],        # staged for A
    "short": [1, 2, 3, 1, 4],                                     # a lane loads its own row
    "long": [12, 9, 700, 10, 11],                                 # one row of 22 segments in five
    "empty": [0, 40, 0, 33],
}


@pytest.mark.parametrize("kind", list(LENGTHS))
@pytest.mark.parametrize("m", [1, 31, 32, 33, 64, 161, 257])
@pytest.mark.parametrize("wide", [3, 11])           # columns per row of A: long and short rows of A^T
def test_residual_of_a_solve(gpu, m, kind, wide):
    sk = gpu
    n = wide * m + 5
    base = LENGTHS[kind]
    lengths = [base[i % len(base)] for i in range(m)]
    if kind == "empty" and m > 64:
        lengths[32:64] = [0] * 32                    # a whole block without entries
    A = _matrix(m, n, lengths, m)
    full = np.asarray(lengths) > 0
    rng = np.random.default_rng(m + 1)
    theta = np.exp(rng.uniform(-1.0, 1.0, n))
    rhs = np.where(full, rng.standard_normal(m), 0.0)
    for prec in (sk.PREC_FP64, sk.PREC_MIXED):
        k = sk.Kkt(m, n, A.indptr.astype(np.int32), A.indices.astype(np.int32), np.ascontiguousarray(A.data),
                   precision=prec)
        assert k.factorize(theta) == 0
        rc, y = k.solve(rhs, tol=1e-11)
        assert rc == 0
        r = rhs - A @ (theta * (A.T @ y))
        assert np.max(np.abs(r)) <= 2e-11 * max(1.0, np.max(np.abs(rhs)))
        k.close()
