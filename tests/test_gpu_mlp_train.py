"""Training's fused launches (gemm_nt_tc_kernel with two products and a bias
gradient, packed epochs, the step's graph) at the sizes where they can go
wrong: batches that are not whole 64-row K chunks or 128-row tiles, layers of
one tile and of several, wide and odd networks, several steps per epoch and a
last partial batch that is dropped.

Gradients: against the numpy oracle with the bars of the network's own test
(3e-3 of each layer's gradient norm, 1e-5 in cosine; they come from
activations that cross a bf16 rounding boundary).  Training: against the same
steps taken one by one, gradients from the library and Adam in numpy, in the
order that std::shuffle gives.  The gradients are then the same bits until a
parameter differs by FP32 rounding in Adam (1e-7 of it), so after three steps
nearly every parameter agrees to a small part of one step, lr."""
import subprocess

import numpy as np
import pytest

from oracle import mlp_oracle
from spacelab_gb300 import surrogate as S

pytestmark = pytest.mark.gpu

ARCHS = [dict(n_in=8, hidden=256, layers=4, n_out=4), dict(n_in=3, hidden=33, layers=1, n_out=5),
         dict(n_in=40, hidden=288, layers=2, n_out=36)]


def _net(arch, max_batch, seed=4):
    return S.Mlp(arch["n_in"], arch["n_out"], arch["hidden"], arch["layers"], max_batch=max_batch, seed=seed)


@pytest.mark.parametrize("arch", ARCHS)
@pytest.mark.parametrize("rows", [32, 96, 160, 1024])
def test_gradients(arch, rows):
    net = _net(arch, 1024)
    rng = np.random.default_rng(rows)
    x = rng.normal(size=(rows, arch["n_in"])).astype(np.float32)
    y = rng.normal(size=(rows, arch["n_out"])).astype(np.float32)
    loss, g = net.gradients(x, y)
    l_ref, g_ref = mlp_oracle.loss_and_grads(net.params(), x, y, **arch)
    assert abs(loss - l_ref) <= 1e-3 * l_ref
    din, dout, offs, _ = mlp_oracle.layout(**arch)
    for (w, b), i, o in zip(offs, din, dout):
        for lo, hi in ((w, w + i * o), (b, b + o)):
            nr = np.linalg.norm(g_ref[lo:hi])
            assert np.linalg.norm(g[lo:hi] - g_ref[lo:hi]) <= 3e-3 * nr
            assert g[lo:hi] @ g_ref[lo:hi] > (1 - 1e-5) * np.linalg.norm(g[lo:hi]) * nr


def _shuffled(n, seed, epochs, tmp_path):
    src = tmp_path / "s.cpp"
    src.write_text('#include <algorithm>\n#include <cstdio>\n#include <random>\n#include <vector>\nint main() {\n'
                   f'std::mt19937_64 rng({seed}); std::vector<int> v({n}); for (int i = 0; i < {n}; ++i) v[i] = i;\n'
                   f'for (int e = 0; e < {epochs}; ++e) {{ std::shuffle(v.begin(), v.end(), rng);\n'
                   'for (int i : v) std::printf("%d ", i); }}\n')
    subprocess.run(["g++", "-O2", str(src), "-o", str(tmp_path / "s")], check=True)
    out = subprocess.run([str(tmp_path / "s")], stdout=subprocess.PIPE, check=True, text=True).stdout
    return np.array(out.split(), dtype=int).reshape(epochs, n)


@pytest.mark.parametrize("arch", ARCHS)
@pytest.mark.parametrize("batch,n,epochs", [(96, 96 * 2 + 31, 2), (128, 128 * 3, 1), (32, 32, 3)])
def test_training_steps(arch, batch, n, epochs, tmp_path):
    lr = 1e-3
    rng = np.random.default_rng(5)
    x = rng.normal(size=(n, arch["n_in"])).astype(np.float32)
    y = rng.normal(size=(n, arch["n_out"])).astype(np.float32)
    net, ref = _net(arch, 128), _net(arch, 128)
    curve = net.train(x, y, epochs=epochs, batch=batch, lr=lr, seed=9)
    p = ref.params().astype(np.float64)
    m, v, t, want = np.zeros_like(p), np.zeros_like(p), 0, []
    for order in _shuffled(n, 9, epochs, tmp_path):
        losses = []
        for k in range(n // batch):
            rows = order[k * batch: (k + 1) * batch]
            loss, g = ref.gradients(x[rows], y[rows])
            losses.append(loss)
            t += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g.astype(np.float64) ** 2
            p = p - lr * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
            ref.set_params(p)
        want.append(np.mean(losses))
    assert np.allclose(curve, want, rtol=1e-3)
    off = np.abs(net.params() - p)
    assert np.quantile(off, 0.99) <= 0.02 * lr and off.max() <= 2 * t * lr
