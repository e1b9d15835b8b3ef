"""A wait in the cooperative training kernel that gives up: the call fails, nothing is trained on what the copy had not
brought, and the network goes on afterwards as if the call had not been made.  (With a limit of no polls the wait gives
up at once; the kernel then waits for the copy itself before it ends.)"""
import numpy as np
import pytest

import jupiterncsm_gb300 as jn

pytestmark = pytest.mark.gpu
TIMEOUT = 7


# some CTAs without samples (37), more than one round of them (1300), a second launch that finds the first one's word (1030 steps)
@pytest.mark.parametrize("n,steps", [(37, 5), (1300, 3), (37, 1030)])
def test_gives_up_before_the_step(n, steps):
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    t = rng.standard_normal((n, 6)).astype(np.float32)
    net, same = (jn.MLP(4, 40, 6, seed=2) for _ in range(2))
    for m in (net, same):
        m.train(x, t, steps=2)
    p = net.params()
    net.set_wait_limit(0)
    for call in (lambda: net.train(x, t, steps=steps), lambda: net.loss_and_gradient(x, t)):
        with pytest.raises(jn.JnError) as e:
            call()
        assert e.value.status == TIMEOUT
        assert np.array_equal(net.params(), p)
    net.set_wait_limit(1 << 20)
    # the moments and the number of steps taken are as they were, too
    assert net.train(x, t, steps=3) == same.train(x, t, steps=3)
    assert np.array_equal(net.params(), same.params())
    assert np.array_equal(net.predict(x), same.predict(x))
    for m in (net, same):
        m.close()


def test_refuses_a_negative_limit():
    net = jn.MLP(2, 4, 2)
    with pytest.raises(jn.JnError):
        net.set_wait_limit(-1)
    net.close()
