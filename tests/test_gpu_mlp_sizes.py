"""The warm start's network at the sizes where its kernels change: tile and chunk remainders, one sample, more samples
than one round of CTAs takes, rows that are no multiple of 16 bytes, networks too wide for shared memory, and more
steps than one launch takes."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn
from oracle import mlp

pytestmark = pytest.mark.gpu
FP32_REL = 1e-4         # FP32 sums against the float64 oracle, relative to the largest magnitude


def _data(seed, n, n_in, n_out):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1, 1, (n, n_in)).astype(np.float32), rng.standard_normal((n, n_out)).astype(np.float32)


@pytest.mark.parametrize("n_in,h,n_out,n", [(1, 4, 1, 1), (3, 17, 5, 16), (4, 128, 32, 256), (4, 129, 33, 257), (8, 160, 40, 300),
                                            (5, 100, 300, 700), (4, 200, 8, 1300), (4, 256, 8, 100), (2, 16, 520, 40)])
def test_forward_and_gradient(n_in, h, n_out, n):
    x, t = _data(h + n, n, n_in, n_out)
    net = jn.MLP(n_in, h, n_out, seed=2)
    p = net.params()
    y_ref, _ = mlp.forward(p, x, n_in, h, n_out)
    assert np.abs(net.predict(x) - y_ref).max() <= FP32_REL * np.abs(y_ref).max()
    loss, g = net.loss_and_gradient(x, t)
    loss_ref, g_ref = mlp.loss_and_gradient(p, x, t, n_in, h, n_out)
    assert abs(loss - loss_ref) <= FP32_REL * loss_ref
    assert np.abs(g - g_ref).max() <= FP32_REL * np.abs(g_ref).max()
    # one Adam step moves every parameter by at most the learning rate, against its gradient
    net.train(x, t, steps=1, learning_rate=1e-3)
    d = net.params() - p
    assert np.abs(d).max() <= 1.001e-3
    big = np.abs(g_ref) > 1e-3 * np.abs(g_ref).max()
    assert np.array_equal(np.sign(d[big]), -np.sign(g_ref[big]))
    net.close()


def test_a_run_split_over_launches_is_the_same_run():
    x, t = _data(4, 37, 4, 6)
    one, two = (jn.MLP(4, 20, 6, seed=7) for _ in range(2))
    loss = one.train(x, t, steps=1030)
    two.train(x, t, steps=1024)
    assert two.train(x, t, steps=6) == loss
    assert np.array_equal(one.params(), two.params())
    one.close()
    two.close()
