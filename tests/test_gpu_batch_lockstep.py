"""The batch's lockstep form (all instances step together, sl_batch.cu) and the
listed close pairs of its mixed tiles, at the batches where they can go wrong:
one instance and one sphere, more instances than CTAs, fewer tiles than warps,
write steps next to each other, runs continued from a later step, and tiles
whose pairs are nearly all close (several list segments).  Exact: bit for bit
the per-sphere loop, which shares no pair code with the tiles.  Mixed: against
the exact batch, with the mixed form's bar of 1e-6 on energies and positions
in radii, over few steps."""
import numpy as np
import pytest

from cases import RADIUS, contact_case
from spacelab_gb300 import BallGroup
from spacelab_gb300 import batch as B

pytestmark = pytest.mark.gpu

STATE = ("pos", "vel", "w", "acc", "aacc")


def _instance(n, seed, spacing=1.97):
    c = contact_case(n, seed, spacing=spacing)
    col = B.Collision(n, 0, 0.0, 0.0, np.sqrt(c["kout"] / c["kin"]), 0.3, seed)
    col.group = BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])
    col.dt, col.kin, col.kout = c["dt"], c["kin"], c["kout"]
    return col


SIZES = {"one": [1], "pair": [2, 1], "few": [33, 64, 95, 300], "many": [5 + (7 * k) % 60 for k in range(400)],
         "uneven": [700, 3, 40, 40]}


def _run(cols, mode, shape, steps, skip, parts=1):
    run = B.BatchRun(cols, mode, steps=steps, skip=skip)
    run.set_shape(*shape)
    per = steps // parts
    for k in range(parts):
        run.run(1 + k * per, per, do_init=k == 0)
    assert not run.status().any()
    out = {**run.state(), "energy": run.energy()}
    run.close()
    return out


@pytest.mark.parametrize("name", sorted(SIZES))
@pytest.mark.parametrize("skip,parts", [(1, 1), (4, 2), (100, 1)])
def test_exact_lockstep(name, skip, parts):
    cols = [_instance(n, 10 + k) for k, n in enumerate(SIZES[name])]
    a = _run(cols, "exact", (0, 128), 8, skip, parts)
    b = _run(cols, "exact", (64, 128), 8, skip, parts)
    for k in STATE:
        assert np.array_equal(a[k], b[k]), k
    scale = np.abs(b["energy"]).max(axis=(1, 2), keepdims=True)
    assert (np.abs(a["energy"] - b["energy"]) <= 1e-10 * scale).all()


@pytest.mark.parametrize("name", sorted(SIZES))
@pytest.mark.parametrize("spacing", [1.97, 1.2])  # 1.2: most pairs of a tile are close
def test_mixed_lockstep(name, spacing):
    cols = [_instance(n, 50 + k, spacing) for k, n in enumerate(SIZES[name])]
    mixed = _run(cols, "mixed_df", (0, 128), 3, 1)
    exact = _run(cols, "exact", (64, 128), 3, 1)
    assert np.abs(mixed["pos"] - exact["pos"]).max() <= 1e-6 * RADIUS
    scale = np.abs(exact["energy"][:, :, :2]).max(axis=(1, 2), keepdims=True)
    assert (np.abs(mixed["energy"] - exact["energy"])[:, :, :2] <= 1e-6 * scale).all()


def test_mixed_lockstep_equals_the_queue():
    """Both forms of the mixed pair-tile pass add the same terms in the same
    order: 512 threads on evenly sized instances take the queue, 128 threads
    on a batch with one large instance lockstep."""
    cols = [_instance(60, 80 + k) for k in range(400)]
    big = _instance(900, 79)
    queue = _run(cols, "mixed_df", (0, 512), 6, 3)
    lock = _run([big] + cols, "mixed_df", (0, 128), 6, 3)
    for k in STATE:
        assert np.array_equal(queue[k], lock[k][900:]), k
