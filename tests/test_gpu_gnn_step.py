"""A training step is over when sk_gnn_train_step returns: parameters read or set right after it,
on other streams than the network's, see the whole step and nothing of it comes later."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def trained(gpu):
    sk = gpu
    m, n = 4000, 30000                       # about a millisecond of gradient behind the loss
    lp = sk.random_lp(m, n, 0.003, 6)
    rp, ci, v = lp.csr()
    rng = np.random.default_rng(6)
    t = (rng.normal(0, 1.5, n), rng.normal(0, 1.5, n), rng.normal(0, 1, m))
    net = sk.Gnn(6)
    bt = sk.GnnBatch.from_arrays(m, n, rp, ci, v, lp.b, lp.c, t)
    yield net, bt
    bt.close()
    net.close()


def test_parameters_read_after_a_step(trained):
    net, bt = trained
    for _ in range(5):
        before = net.get_params()
        net.train_step(bt, 1e-3)
        at_once = net.get_params()
        net.loss_grad(bt)                    # waits for the network's stream
        np.testing.assert_array_equal(at_once, net.get_params())
        assert np.max(np.abs(at_once - before)) > 0.0


def test_parameters_set_after_a_step(trained):
    net, bt = trained
    p = net.get_params()
    for _ in range(5):
        net.train_step(bt, 1e-3)
        net.set_params(p)
        net.loss_grad(bt)
        np.testing.assert_array_equal(net.get_params(), p)
