"""The learned-start network's kernels at the edges of their node tiles (16 and 32 nodes) and of
the rule between them, against the FP64 oracle on BF16 weights; the bounds are those of FP32
accumulation over 64 features and a few layers, as for the smaller graphs."""
import numpy as np
import pytest

import gnn_oracle as go

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,d", [(3, 5, 0.9), (15, 33, 0.3), (16, 32, 0.3), (17, 257, 0.1),
                                   (31, 9727, 0.05), (33, 9729, 0.05)])
def test_prediction_and_gradient(gpu, m, n, d):
    sk = gpu
    lp = sk.random_lp(m, n, d, 9)
    rp, ci, v = lp.csr()
    rng = np.random.default_rng(m)
    t = (rng.normal(0, 1.5, n), rng.normal(0, 1.5, n), rng.normal(0, 1, m))
    p = go.glorot_params(9)
    net = sk.Gnn(9)
    net.set_params(p)
    bt = sk.GnnBatch.from_arrays(m, n, rp, ci, v, lp.b, lp.c, t)
    rx, rs, ry, rloss, cache = go.forward(p, m, n, rp, ci, v, lp.b, lp.c, t, bf16=True)
    for a, r in zip(net.predict(bt), (rx, rs, ry)):
        assert np.max(np.abs(a - r)) <= 1e-4 * (1.0 + np.max(np.abs(r)))
    loss, g = net.loss_grad(bt)
    rg = go.backward(cache)
    assert abs(loss - rloss) <= 1e-5 * rloss
    assert np.linalg.norm(g - rg) <= 1e-3 * np.linalg.norm(rg)
    bt.close()
    net.close()
