"""The network's two paths give the same bits: the cooperative kernel (weights in shared memory) and the kernels a pass
(networks too wide for it).  A narrow network is run by the second path as part of a wide one whose other units have
zero weights: they add exact zeros to every sum, and their gradients are zero, so they stay zero."""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn

pytestmark = pytest.mark.gpu
WIDE = 256              # 256 x 256 weights are above the shared memory of an SM


def _parts(p, n_in, h, n_out):
    """W1, b1, W2, b2, W3, b3 of a parameter array."""
    shapes, out, at = [(h, n_in), (h,), (h, h), (h,), (n_out, h), (n_out,)], [], 0
    for s in shapes:
        n = int(np.prod(s))
        out.append(p[at:at + n].reshape(s))
        at += n
    assert at == len(p)
    return out


def _widened(p, n_in, h, n_out):
    wide = [np.zeros(s, np.float32) for s in [(WIDE, n_in), (WIDE,), (WIDE, WIDE), (WIDE,), (n_out, WIDE), (n_out,)]]
    for a, b in zip(wide, _parts(p, n_in, h, n_out)):
        a[tuple(slice(n) for n in b.shape)] = b
    return np.concatenate([a.reshape(-1) for a in wide])


# one sample a CTA, two, four and eight with remainders; rows that are no multiple of 16 bytes; one unit; 128 and 160
# units, whose shares of the weights are uneven numbers of rows
@pytest.mark.parametrize("n_in,h,n_out,n", [(1, 1, 1, 1), (3, 17, 5, 16), (4, 128, 32, 256), (4, 129, 33, 153), (8, 160, 40, 300),
                                            (5, 100, 250, 607), (6, 33, 9, 1300)])
def test_same_bits(n_in, h, n_out, n):
    rng = np.random.default_rng(h + n)
    x = rng.uniform(-1, 1, (n, n_in)).astype(np.float32)
    t = rng.standard_normal((n, n_out)).astype(np.float32)
    a, b = jn.MLP(n_in, h, n_out, seed=3), jn.MLP(n_in, WIDE, n_out)
    p = a.params()
    b.set_params(_widened(p, n_in, h, n_out))
    assert np.array_equal(a.predict(x), b.predict(x))
    (la, ga), (lb, gb) = a.loss_and_gradient(x, t), b.loss_and_gradient(x, t)
    assert la == lb
    assert np.array_equal(_widened(ga, n_in, h, n_out), gb)
    assert a.train(x, t, steps=7) == b.train(x, t, steps=7)
    assert np.array_equal(_widened(a.params(), n_in, h, n_out), b.params())
    assert np.array_equal(a.predict(x), b.predict(x))
    a.close()
    b.close()
