"""The steps of a dense factorisation (diagonal tile, panel, trailing update, on the FP64 pipe
and with BF16 digits) and the triangular solves at the edges of their tiles, parts and rules,
against FP64 numpy.

A factor is checked through L L^T = D A Theta A^T D + delta I. Standard error analysis bounds
an entry's error by (m + 1) u (|L| |L^T|)_ij <= (m + 1) u (1 + delta); the panel is multiplied by
the inverse of the 64 x 64 diagonal tile, which adds 64 u times |Linv| |L| of the worst tile, and
the digits of the emulated path add at most m u / 2 (rows to 2^-56 of their largest entry)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
DELTA = 1e-9


def _system(m, n, seed, per_col=8):
    rng = np.random.default_rng(seed)
    A = np.zeros((m, n))
    for j in range(n):
        r = rng.choice(m, size=min(m, per_col), replace=False)
        A[r, j] = rng.standard_normal(r.size)
    A[:, :m] += 2.0 * np.eye(m)
    return A, np.exp(rng.uniform(-1.0, 1.0, n)), rng.standard_normal(m)


def _kkt(sk, A, mode=None, precision=None):
    m, n = A.shape
    rp = np.concatenate(([0], np.cumsum((A != 0).sum(1)))).astype(np.int32)
    ci = np.nonzero(A)[1].astype(np.int32)
    k = sk.Kkt(m, n, rp, ci, np.ascontiguousarray(A[A != 0]), P=np.arange(m, dtype=np.int32),
               precision=sk.PREC_FP64 if precision is None else precision)
    if mode is not None:
        k.set_fp64_update(mode)
    return k


def _check_factor(k, A, theta):
    m = A.shape[0]
    L, D = k.factor_dense()
    M = (A * theta) @ A.T
    M = M * D[:, None] * D[None, :] + DELTA * np.eye(m)
    L0 = np.linalg.cholesky(M)
    tile = 1.0
    for b in range(0, m, 64):
        T = L0[b:b + 64, b:b + 64]
        tile = max(tile, np.max((np.abs(np.linalg.inv(T)) @ np.abs(T)).sum(1)))
    err = np.max(np.abs(np.tril(L) @ np.tril(L).T - M))
    assert err <= (2 * m + 2 + 128 * tile) * U * (1.0 + DELTA), (m, err / U, tile)


def _check_solve(k, A, theta, rhs, tol):
    rc, y = k.solve(rhs, tol=tol)
    assert rc == 0
    r = rhs - A @ (theta * (A.T @ y))
    assert np.max(np.abs(r)) <= 2.0 * tol * max(1.0, np.max(np.abs(rhs)))


# tiles and remainders; 16 and 32 parts (24 tiles), the diagonal tile alone on its SM (300)
@pytest.mark.parametrize("tensor", [False, True])
@pytest.mark.parametrize("m", [1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 193, 320, 511, 1665])
def test_factor_and_solve(gpu, m, tensor):
    sk = gpu
    A, theta, rhs = _system(m, 2 * m + 5, m, per_col=4 if m > 200 else 8)
    k = _kkt(sk, A, sk.FP64_UPDATE_TENSOR if tensor else sk.FP64_UPDATE_NATIVE)
    assert k.factorize(theta) == 0
    _check_factor(k, A, theta)
    _check_solve(k, A, theta, rhs, 1e-12)
    k.close()


@pytest.mark.parametrize("m", [1, 16, 65, 129, 1100])
def test_mixed_solve(gpu, m):
    sk = gpu
    A, theta, rhs = _system(m, 2 * m + 5, m + 7, per_col=4)
    k = _kkt(sk, A, precision=sk.PREC_MIXED)
    assert k.factorize(theta) == 0
    _check_solve(k, A, theta, rhs, 1e-9)
    k.close()


# Rows whose panel entries are near 2^-964 beside ordinary ones: the digits' scales leave the
# normal range in some rows of a warp's 32 and not in others.
@pytest.mark.parametrize("m", [200, 330])
def test_rows_of_tiny_entries(gpu, m):
    sk = gpu
    A, theta, rhs = _system(m, 2 * m + 5, 3)
    tiny = np.arange(m) % 3 == 1
    tiny[:128] = False
    A[tiny] *= 1e-290
    A[tiny, np.arange(m)[tiny]] = 2.0
    A[~tiny, :] *= np.where(np.isin(np.arange(A.shape[1]), np.arange(m)[tiny]), 0.0, 1.0)
    k = _kkt(sk, A, sk.FP64_UPDATE_TENSOR)
    assert k.factorize(theta) == 0
    _check_factor(k, A, theta)
    _check_solve(k, A, theta, rhs, 1e-12)
    k.close()


# A pivot that is not a number ends the factorisation at any place of a tile, and only that one.
@pytest.mark.parametrize("mode", ["native", "tensor", "mixed"])
@pytest.mark.parametrize("row", [0, 5, 16, 63, 64, 100, 149])
def test_bad_pivot(gpu, row, mode):
    sk = gpu
    A, theta, rhs = _system(150, 305, 11)
    prec = sk.PREC_MIXED if mode == "mixed" else sk.PREC_FP64
    k = _kkt(sk, A, sk.FP64_UPDATE_TENSOR if mode == "tensor" else sk.FP64_UPDATE_NATIVE, prec)
    bad = theta.copy()
    bad[row] = np.nan
    assert k.factorize(bad) != 0
    assert k.factorize(theta) == 0
    _check_solve(k, A, theta, rhs, 1e-9)
    k.close()
