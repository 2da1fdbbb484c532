"""A surrogate call that goes wrong is reported or done another way, and the
next one does not suffer from it: a prediction in place that meets a slow page
of host memory, a rejected launch, a call whose wait ran out.  The failures are
made on the host (sl_diag_mlp_fail), as is a product that cannot be set up; results bit for bit those of an untroubled
call."""
import numpy as np
import pytest

from spacelab_gb300 import _lib
from spacelab_gb300 import surrogate as S
from spacelab_gb300._lib import check

pytestmark = pytest.mark.gpu

SLOW_PAGE, LAUNCH, TIMED_OUT, SETUP = 1, 2, 3, 4


@pytest.fixture(scope="module")
def net():
    return S.Mlp(8, 4, 64, 2, max_batch=128, seed=2)


def _x(n):
    return np.random.default_rng(n).normal(size=(n, 8)).astype(np.float32)


def _fail(net, what):
    check(net.lib.sl_diag_mlp_fail(net.h, what), "sl_diag_mlp_fail")


@pytest.mark.parametrize("n", [1, 128, 500])
def test_a_slow_page(net, n):
    want = net.predict(_x(n))
    _fail(net, SLOW_PAGE)
    assert np.array_equal(net.predict(_x(n)), want)
    assert np.array_equal(net.predict(_x(n)), want)


def test_a_rejected_launch(net):
    want = net.predict(_x(100))
    _fail(net, LAUNCH)
    with pytest.raises(_lib.SpaceLabError) as err:
        net.predict(_x(100))
    assert err.value.code == _lib.SL_ERR_CUDA
    assert np.array_equal(net.predict(_x(100)), want)


def test_calls_after_one_that_timed_out(net):
    x, y = _x(64), _x(64)[:, :4]
    want, (loss, grads) = net.predict(x), net.gradients(x, y)
    _fail(net, TIMED_OUT)
    assert np.array_equal(net.predict(x), want)
    _fail(net, TIMED_OUT)
    l2, g2 = net.gradients(x, y)
    assert l2 == loss and np.array_equal(g2, grads)
    _fail(net, TIMED_OUT)
    assert np.isfinite(net.train(x, y, epochs=1, batch=32)).all()


def test_training_without_a_product_changes_nothing():
    x, y = _x(64), _x(64)[:, :4]
    a, b = (S.Mlp(8, 4, 64, 2, max_batch=128, seed=5) for _ in range(2))
    a.gradients(x, y)  # gradients that a step must not take
    before = a.params()
    _fail(a, SETUP)
    with pytest.raises(_lib.SpaceLabError) as err:
        a.train(x, y, epochs=1, batch=32)
    assert err.value.code == _lib.SL_ERR_CUDA
    assert np.array_equal(a.params(), before)
    assert np.array_equal(a.train(x, y, epochs=2, batch=32), b.train(x, y, epochs=2, batch=32))
    assert np.array_equal(a.params(), b.params())
