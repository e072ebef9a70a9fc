"""Factorisations large or numerous enough for the steady state of the step kernels, entry by
entry: one dense front from which a block of the emulated-FP64 update takes runs of tiles (its
buffers and its ring of tiles are used again, rows of A stay over a run) and the FP64 panel solve
16 rows a block; and more fronts than SMs, so that one block factors two diagonal tiles a step.

An entry of L L^T is off by at most (m + 1) u (|L| |L^T|)_ij <= (m + 1) u (1 + delta) from the sums
(m: rows of the front), 64 u |Linv| |L| of the worst 64 x 64 tile from the panel solve and
m u / 2 from the digits of the emulated path."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
DELTA = 1e-9


def _block(m, seed, per_col=6):
    """m x 2m, six entries a column and one dense column, so that the normal matrix is full."""
    rng = np.random.default_rng(seed)
    n = 2 * m
    rows = rng.integers(0, m, (n, per_col))
    A = sp.csr_matrix((rng.standard_normal(rows.size), (rows.ravel(), np.repeat(np.arange(n), per_col))), (m, n))
    A = A + sp.eye(m, n) * 3.0
    dense = sp.csr_matrix(0.05 + 0.05 * rng.random((m, 1)))
    return sp.hstack([A, dense]).tocsr()


def _kkt(sk, A, mode, P=None):
    A.sum_duplicates()
    A.sort_indices()
    k = sk.Kkt(A.shape[0], A.shape[1], A.indptr.astype(np.int32), A.indices.astype(np.int32),
               np.ascontiguousarray(A.data), P=P)
    k.set_fp64_update(sk.FP64_UPDATE_TENSOR if mode == "tensor" else sk.FP64_UPDATE_NATIVE)
    return k


def _check(L, D, A, theta):
    m = A.shape[0]
    M = (A.multiply(theta) @ A.T).toarray()
    M = M * D[:, None] * D[None, :] + DELTA * np.eye(m)
    L = np.tril(L)
    tile = 1.0
    for b in range(0, m, 64):
        T = L[b:b + 64, b:b + 64]
        tile = max(tile, np.max((np.abs(np.linalg.inv(T)) @ np.abs(T)).sum(1)))
    err = np.max(np.abs(L @ L.T - M))
    assert err <= (2 * m + 2 + 128 * tile) * U * (1.0 + DELTA), (m, err / U, tile)


# 3600 rows: runs of 2 tiles; 4993: runs of 4, and 77 panel units of 64 rows
@pytest.mark.parametrize("m,mode", [(3600, "tensor"), (4993, "tensor"), (4993, "native")])
def test_one_large_front(gpu, m, mode):
    A = _block(m, m)
    theta = np.exp(np.random.default_rng(1).uniform(-1.0, 1.0, A.shape[1]))
    k = _kkt(gpu, A, mode)
    assert k.factorize(theta) == 0
    L, D = k.factor_dense()
    _check(L, D, A, theta)
    rhs = np.random.default_rng(2).standard_normal(m)
    rc, y = k.solve(rhs, tol=1e-12)
    assert rc == 0
    assert np.max(np.abs(rhs - A @ (theta * (A.T @ y)))) <= 2e-12 * max(1.0, np.max(np.abs(rhs)))
    k.close()


# 11 fronts of about 700 rows (110 panel units and 330 tiles of 128 x 64 in the first step), and
# 170 fronts of 65 to 130 rows (more first tiles than SMs)
@pytest.mark.parametrize("mode", ["native", "tensor"])
@pytest.mark.parametrize("sizes", [[700, 641, 703, 768, 690, 705, 640, 767, 699, 701, 720],
                                   [65 + (37 * q) % 66 for q in range(170)]], ids=["eleven", "many"])
def test_several_fronts(gpu, sizes, mode):
    blocks = [_block(m, 100 + q) for q, m in enumerate(sizes)]
    A = sp.block_diag(blocks).tocsr()
    m = A.shape[0]
    theta = np.exp(np.random.default_rng(3).uniform(-1.0, 1.0, A.shape[1]))
    k = _kkt(gpu, A, mode, P=np.arange(m, dtype=np.int32))
    assert k.factorize(theta) == 0
    L, D = k.factor_dense()
    r0 = c0 = 0
    for B in blocks:
        r1, c1 = r0 + B.shape[0], c0 + B.shape[1]
        _check(L[r0:r1, r0:r1], D[r0:r1], B, theta[c0:c1])
        r0, c0 = r1, c1
    rhs = np.random.default_rng(4).standard_normal(m)
    rc, y = k.solve(rhs, tol=1e-12)
    assert rc == 0
    assert np.max(np.abs(rhs - A @ (theta * (A.T @ y)))) <= 2e-12 * max(1.0, np.max(np.abs(rhs)))
    k.close()
