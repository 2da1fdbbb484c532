"""A surrogate call that goes wrong is reported, and the next one does not
suffer from it: a rejected launch.  The failure is made on the host
(sl_diag_mlp_fail); results bit for bit those of an untroubled call."""
import numpy as np
import pytest

from spacelab_gb300 import _lib
from spacelab_gb300 import surrogate as S
from spacelab_gb300._lib import check

pytestmark = pytest.mark.gpu

LAUNCH = 2


@pytest.fixture(scope="module")
def net():
    return S.Mlp(8, 4, 64, 2, max_batch=128, seed=2)


def _x(n):
    return np.random.default_rng(n).normal(size=(n, 8)).astype(np.float32)


def _fail(net, what):
    check(net.lib.sl_diag_mlp_fail(net.h, what), "sl_diag_mlp_fail")


def test_a_rejected_launch(net):
    want = net.predict(_x(100))
    _fail(net, LAUNCH)
    with pytest.raises(_lib.SpaceLabError) as err:
        net.predict(_x(100))
    assert err.value.code == _lib.SL_ERR_CUDA
    assert np.array_equal(net.predict(_x(100)), want)
