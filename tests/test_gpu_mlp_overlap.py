"""Predictions written over their inputs (fewer outcomes than features, so that
a batch's results never reach a later batch's rows), against separate arrays,
bit for bit: one tile, several, more tiles than CTAs, one batch and many."""
import ctypes

import numpy as np
import pytest

from spacelab_gb300 import surrogate as S
from spacelab_gb300._lib import check

pytestmark = pytest.mark.gpu

_fp = ctypes.POINTER(ctypes.c_float)


@pytest.mark.parametrize("n_out", [1, 7, 8])
@pytest.mark.parametrize("n", [100, 1000, 152 * 128 * 5 + 3])
def test_results_over_inputs(n, n_out):
    net = S.Mlp(8, n_out, 64, 2, max_batch=256, seed=3)
    x = np.random.default_rng(n).normal(size=(n, 8)).astype(np.float32)
    want = net.predict(x)
    p = x.ctypes.data_as(_fp)
    check(net.lib.sl_mlp_predict(net.h, p, n, p), "sl_mlp_predict")
    assert np.array_equal(x.reshape(-1)[: n * n_out].reshape(n, n_out), want)
