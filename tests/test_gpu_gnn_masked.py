"""A masked gradient (exactly 0) leaves its node out of the weight gradients, whatever that
node's features and activations are: a NaN or an infinity there takes nothing from the other
nodes. Against the FP64 oracle on BF16 weights, with the bounds of the finite graphs
(FP32 accumulation over 64 features and a few layers)."""
import numpy as np
import pytest

import gnn_oracle as go

pytestmark = pytest.mark.gpu
SIZES = [(40, 90, 0.1), (33, 9729, 0.05)]


def _graph(sk, m, n, d):
    lp = sk.random_lp(m, n, d, 4)
    rp, ci, v = lp.csr()
    rng = np.random.default_rng(n)
    t = (rng.normal(0, 1.5, n), rng.normal(0, 1.5, n), rng.normal(0, 1, m))
    return rp, ci, v, np.array(lp.b), np.array(lp.c), t


def _gradient(sk, p, m, n, rp, ci, v, b, c, t):
    net = sk.Gnn(1)
    net.set_params(p)
    bt = sk.GnnBatch.from_arrays(m, n, rp, ci, v, b, c, t)
    loss, g = net.loss_grad(bt)
    bt.close()
    net.close()
    return loss, g


def _check(loss, g, rloss, rg):
    assert np.isfinite(loss) and np.all(np.isfinite(g))
    assert abs(loss - rloss) <= 1e-5 * rloss
    for name, (o, s) in go.layout()[0].items():
        k = int(np.prod(s))
        ref = rg[o:o + k]
        assert np.linalg.norm(g[o:o + k] - ref) <= 2e-3 * np.linalg.norm(rg) + 1e-3 * np.linalg.norm(ref), name


@pytest.mark.parametrize("m,n,d", SIZES)
def test_feature_that_is_no_number(gpu, monkeypatch, m, n, d):
    rp, ci, v, b, c, t = _graph(gpu, m, n, d)
    b[m // 2] = c[n // 3] = c[n - 1] = np.nan          # embeddings of 0: NaN > 0 is false
    p = go.glorot_params(2)
    monkeypatch.setattr(go, "_relu", lambda x: np.where(x > 0, x, 0.0))
    _, _, _, rloss, cache = go.forward(p, m, n, rp, ci, v, b, c, t)
    for f in ("fr", "fc"):
        cache[f] = np.nan_to_num(cache[f])             # met by gradients of 0 alone
    _check(*_gradient(gpu, p, m, n, rp, ci, v, b, c, t), rloss, go.backward(cache))


# One column's right-hand side overflows in FP32: its feature K is infinite, every other one 0,
# and so are its rows' messages; the next layer's weights of that feature are negative, so that
# its nodes there are masked.
@pytest.mark.parametrize("m,n,d", SIZES)
def test_infinite_activation(gpu, m, n, d):
    rp, ci, v, b, c, t = _graph(gpu, m, n, d)
    c[n // 3] = 1e300
    v = np.where(np.asarray(ci) == n // 3, np.abs(v), v)
    K, p = 5, go.glorot_params(3)
    lay = go.layout()[0]
    E = p[lay["Ec"][0]:][:go.H * 3].reshape(go.H, 3)
    E[:, 0] = -np.abs(E[:, 0]) - 0.125
    E[K, 0] = 0.5
    for W in ("Wcc0", "Wrm0"):
        w = p[lay[W][0]:][:go.H * go.H].reshape(go.H, go.H)
        w[:, K] = -np.abs(w[:, K]) - 0.125
    _, _, _, rloss, cache = go.forward(p, m, n, rp, ci, v, b, c, t)
    _check(*_gradient(gpu, p, m, n, rp, ci, v, b, c, t), rloss, go.backward(cache))
