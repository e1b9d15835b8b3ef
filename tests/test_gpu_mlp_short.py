"""One pass of a small network runs as the kernels of a pass, which start sooner than the cooperative launch.  With a
limit of no polls the cooperative kernel's wait gives up, so a call that succeeds has not taken it; and the other side
of each line does take it."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn

pytestmark = pytest.mark.gpu


def _net(n_in, h, n_out, n):
    rng = np.random.default_rng(h)
    net = jn.MLP(n_in, h, n_out, seed=4)
    x = rng.uniform(-1, 1, (n, n_in)).astype(np.float32)
    return net, x, rng.standard_normal((n, n_out)).astype(np.float32)


@pytest.mark.parametrize("n_in,h,n_out,n,short", [
    (2, 8, 4, 20000, True), (4, 16, 8, 1, True), (4, 32, 8, 1489, True), (4, 32, 8, 1490, False), (4, 128, 32, 64, True),
    (4, 128, 32, 256, False), (8, 160, 40, 1, False)])
def test_predict(n_in, h, n_out, n, short):
    net, x, _ = _net(n_in, h, n_out, n)
    want = net.predict(x)
    net.set_wait_limit(0)
    if short:
        assert np.array_equal(net.predict(x), want)
    else:
        with pytest.raises(jn.JnError):
            net.predict(x)
    net.close()


@pytest.mark.parametrize("n_in,h,n_out,n,short", [(4, 16, 8, 1, True), (4, 32, 8, 32, True), (4, 32, 8, 33, False),
                                                  (4, 64, 16, 1, False)])
def test_gradient(n_in, h, n_out, n, short):
    net, x, t = _net(n_in, h, n_out, n)
    loss, g = net.loss_and_gradient(x, t)
    net.set_wait_limit(0)
    if short:
        again = net.loss_and_gradient(x, t)
        assert again[0] == loss and np.array_equal(again[1], g)
    else:
        with pytest.raises(jn.JnError):
            net.loss_and_gradient(x, t)
    net.close()
