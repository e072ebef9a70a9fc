"""A Newton solve whose residual has an entry that is not finite is no success: the contract is
max |rhs - M y| <= tol max(1, max |rhs|), which a NaN does not meet. The handle solves the next
right-hand side as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SK_ERR_NUMERICAL = 3


def _system(m, seed):
    rng = np.random.default_rng(seed)
    n = 2 * m + 3
    A = np.where(rng.random((m, n)) < min(1.0, 6.0 / n), rng.standard_normal((m, n)), 0.0)
    A[:, :m] += 2.0 * np.eye(m)
    return A, np.exp(rng.uniform(-1.0, 1.0, n)), rng.standard_normal(m)


def _kkt(sk, A, mode):
    m, n = A.shape
    rp = np.concatenate(([0], np.cumsum((A != 0).sum(1)))).astype(np.int32)
    ci = np.nonzero(A)[1].astype(np.int32)
    k = sk.Kkt(m, n, rp, ci, np.ascontiguousarray(A[A != 0]),
               precision=sk.PREC_MIXED if mode == "mixed" else sk.PREC_FP64)
    if mode != "mixed":
        k.set_fp64_update(sk.FP64_UPDATE_TENSOR if mode == "tensor" else sk.FP64_UPDATE_NATIVE)
    return k


def _good(k, A, theta, rhs, tol):
    rc, y = k.solve(rhs, tol=tol)
    assert rc == 0
    r = rhs - A @ (theta * (A.T @ y))
    assert np.max(np.abs(r)) <= 2.0 * tol * max(1.0, np.max(np.abs(rhs)))


@pytest.mark.parametrize("mode", ["native", "tensor", "mixed"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("m", [1, 33, 200])
def test_right_hand_side_that_is_not_finite(gpu, m, bad, mode):
    A, theta, rhs = _system(m, m)
    k = _kkt(gpu, A, mode)
    assert k.factorize(theta) == 0
    for row in sorted({0, m // 2, m - 1}):
        r = rhs.copy()
        r[row] = bad
        rc, _ = k.solve(r, tol=1e-9)
        assert rc == SK_ERR_NUMERICAL, row
    _good(k, A, theta, rhs, 1e-9)
    k.close()


# Rows without a common column: a bad entry reaches one row's solution and no other's.
@pytest.mark.parametrize("mode", ["native", "mixed"])
def test_one_row_that_is_not_finite(gpu, mode):
    m = 150
    A, theta = np.diag(np.linspace(1.0, 2.0, m)), np.linspace(0.5, 1.5, m)
    rhs = np.linspace(-1.0, 1.0, m)
    k = _kkt(gpu, A, mode)
    assert k.factorize(theta) == 0
    r = rhs.copy()
    r[77] = np.nan
    assert k.solve(r, tol=1e-9)[0] == SK_ERR_NUMERICAL
    _good(k, A, theta, rhs, 1e-9)
    k.close()


# 1e39 is beyond the FP32 fronts of the mixed mode, and an ordinary number for FP64 ones.
def test_beyond_the_fronts_range(gpu):
    A, theta, rhs = _system(100, 5)
    rhs[3] = 1e39
    k = _kkt(gpu, A, "mixed")
    assert k.factorize(theta) == 0
    assert k.solve(rhs, tol=1e-9)[0] == SK_ERR_NUMERICAL
    k.close()
    k = _kkt(gpu, A, "native")
    assert k.factorize(theta) == 0
    _good(k, A, theta, rhs, 1e-9)
    k.close()


def test_device_right_hand_side(gpu):
    import torch
    A, theta, rhs = _system(90, 8)
    k = _kkt(gpu, A, "native")
    assert k.factorize(theta) == 0
    d = torch.tensor(rhs, device="cuda")
    d[40] = float("nan")
    torch.cuda.synchronize()
    assert gpu.lib().sk_kkt_solve_device(k.h, d.data_ptr(), 1e-9) == SK_ERR_NUMERICAL
    d = torch.tensor(rhs, device="cuda")
    torch.cuda.synchronize()
    assert gpu.lib().sk_kkt_solve_device(k.h, d.data_ptr(), 1e-9) == 0
    k.close()
