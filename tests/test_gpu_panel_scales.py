"""Panel rows of the emulated-FP64 factorisation whose scales leave the normal range in some of a
warp's 32 rows and not in others (rows near 2^-964, rows without a coupling, padded rows): the
ordinary rows beside them keep the bound of an FP64 factor.

An entry of L L^T is off by at most (m + 1) u (|L| |L^T|)_ij <= (m + 1) u (1 + delta) from the sums,
64 u |Linv| |L| of the worst 64 x 64 tile from the panel solve and m u / 2 from the digits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
DELTA = 1e-9


@pytest.mark.parametrize("pattern", ["one", "odd", "half", "last", "zero"])
@pytest.mark.parametrize("m", [193, 330, 449])
def test_scales_within_a_warp(gpu, m, pattern):
    sk = gpu
    rng = np.random.default_rng(m)
    n = 2 * m + 5
    A = np.zeros((m, n))
    for j in range(n):
        r = rng.choice(m, size=8, replace=False)
        A[r, j] = rng.standard_normal(r.size)
    A[:, :m] += 2.0 * np.eye(m)
    lane = np.arange(m) % 32
    tiny = {"one": lane == 5, "odd": lane % 2 == 1, "half": lane >= 16, "last": lane == 31, "zero": lane % 3 == 0}[pattern]
    tiny[:64] = False
    A[tiny] = 0.0
    own = np.arange(m)[tiny]
    A[:, own] = 0.0
    A[own, own] = 2.0
    if pattern != "zero":                  # coupled to the first 64 rows, by 1e-290 and less
        A[:64, own] = 1e-290 * rng.standard_normal((64, own.size))
    theta, rhs = np.exp(rng.uniform(-1.0, 1.0, n)), rng.standard_normal(m)
    rp = np.concatenate(([0], np.cumsum((A != 0).sum(1)))).astype(np.int32)
    k = sk.Kkt(m, n, rp, np.nonzero(A)[1].astype(np.int32), np.ascontiguousarray(A[A != 0]),
               P=np.arange(m, dtype=np.int32))
    k.set_fp64_update(sk.FP64_UPDATE_TENSOR)
    assert k.factorize(theta) == 0
    L, D = k.factor_dense()
    M = (A * theta) @ A.T
    M = M * D[:, None] * D[None, :] + DELTA * np.eye(m)
    L0 = np.linalg.cholesky(M)
    tile = 1.0
    for b in range(0, m, 64):
        T = L0[b:b + 64, b:b + 64]
        tile = max(tile, np.max((np.abs(np.linalg.inv(T)) @ np.abs(T)).sum(1)))
    err = np.max(np.abs(np.tril(L) @ np.tril(L).T - M))
    assert err <= (2 * m + 2 + 128 * tile) * U * (1.0 + DELTA), (err / U, tile)
    rc, y = k.solve(rhs, tol=1e-12)
    assert rc == 0
    assert np.max(np.abs(rhs - A @ (theta * (A.T @ y)))) <= 2e-12 * max(1.0, np.max(np.abs(rhs)))
    k.close()
