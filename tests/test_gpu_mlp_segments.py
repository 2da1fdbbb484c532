"""Training on a data set larger than the device memory kept for it, in segments
that the host gathers: 600,000 rows of 100 features (570 MB with the packed
epoch, 256 MB kept).  92 of the features are zero, so the network of the other
8, whose 118 MB are trained on whole, takes the same steps: their weights and
losses are the same bits."""
import numpy as np
import pytest

from oracle import mlp_oracle
from spacelab_gb300 import surrogate as S

pytestmark = pytest.mark.gpu


def test_segments_take_the_same_steps():
    torch = pytest.importorskip("torch")
    n, batch = 600_000, 1024
    rng = np.random.default_rng(1)
    x = np.zeros((n, 100), dtype=np.float32)
    x[:, :8] = rng.normal(size=(n, 8))
    y = rng.normal(size=(n, 4)).astype(np.float32)
    small, wide = (S.Mlp(k, 4, 32, 1, max_batch=batch, seed=6) for k in (8, 100))
    (w_s, _), (w_w, _) = (mlp_oracle.layout(n_in=k, hidden=32, layers=1, n_out=4)[2][0] for k in (8, 100))
    p, q = small.params(), np.zeros(wide.num_params(), dtype=np.float32)
    q[w_w: w_w + 32 * 128].reshape(32, 128)[:, :32] = p[w_s: w_s + 32 * 32].reshape(32, 32)
    q[w_w + 32 * 128:] = p[w_s + 32 * 32:]
    wide.set_params(q)
    a = small.train(x[:, :8], y, epochs=2, batch=batch, lr=1e-3, seed=3)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    b = wide.train(x, y, epochs=2, batch=batch, lr=1e-3, seed=3)
    assert free - torch.cuda.mem_get_info()[0] < 300 << 20
    assert np.array_equal(a, b)
    p, q = small.params(), wide.params()
    assert np.array_equal(q[w_w: w_w + 32 * 128].reshape(32, 128)[:, :32], p[w_s: w_s + 32 * 32].reshape(32, 32))
    assert not q[w_w: w_w + 32 * 128].reshape(32, 128)[:, 32:].any()
    assert np.array_equal(q[w_w + 32 * 128:], p[w_s + 32 * 32:])
