"""The one-launch forward pass (mlp_forward_kernel) and the layer-by-layer
one behind it, against the numpy oracle at the sizes where they can go wrong:
row tiles of 128 and their remainders, more tiles than CTAs, widths below and
across the 64-column K chunks and the 128-column weight tiles, one and many
layers, odd feature and outcome counts (no 16-byte groups), inputs that start
off a 16-byte boundary, and networks too wide or too deep for one launch.

Bar: the two sides differ in FP32 accumulation order only, which can move an
activation across a bf16 rounding boundary, one part in 2^8 of it; a layer in
which every unit moved the same way would shift the outputs by 2^-8 of their
scale, so `layers` of them by layers 2^-8."""
import numpy as np
import pytest

from oracle import mlp_oracle
from spacelab_gb300 import surrogate as S

pytestmark = pytest.mark.gpu

NET = dict(n_in=8, hidden=256, layers=4, n_out=4)


def _check(arch, x, net=None):
    net = net or S.Mlp(arch["n_in"], arch["n_out"], arch["hidden"], arch["layers"], max_batch=256, seed=2)
    p = net.params()
    rng = np.random.default_rng(7)
    for (w, b), n in zip(mlp_oracle.layout(**arch)[2], [arch["hidden"]] * arch["layers"] + [arch["n_out"]]):
        p[b: b + n] = rng.normal(0, 0.3, n).astype(np.float32)  # biases, which start at 0
    net.set_params(p)
    y = net.predict(x)
    ref = mlp_oracle.forward(p, x, **arch)[0]
    assert y.shape == ref.shape
    assert np.abs(y - ref).max() <= arch["layers"] * 2.0 ** -8 * np.abs(ref).max()


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 1000, 2 * 152 * 128 + 1])
def test_rows(n):
    x = np.random.default_rng(n).normal(size=(n, 8)).astype(np.float32)
    _check(NET, x)


@pytest.mark.parametrize("arch", [
    dict(n_in=1, hidden=1, layers=1, n_out=1), dict(n_in=3, hidden=33, layers=2, n_out=5),
    dict(n_in=40, hidden=96, layers=3, n_out=7), dict(n_in=100, hidden=160, layers=7, n_out=36),
    dict(n_in=256, hidden=256, layers=1, n_out=256),
    dict(n_in=8, hidden=288, layers=2, n_out=4), dict(n_in=8, hidden=64, layers=8, n_out=4)])
def test_shapes(arch):
    x = np.random.default_rng(3).normal(size=(300, arch["n_in"])).astype(np.float32)
    _check(arch, x)


def test_unaligned_rows():
    buf = np.random.default_rng(4).normal(size=200 * 8 + 1).astype(np.float32)
    x = buf[1:].reshape(200, 8)
    assert x.ctypes.data % 16 != 0
    _check(NET, x)
