"""A batch whose lockstep launch is refused (fewer SMs than CTAs) runs its
per-CTA form instead, with the same state, bit for bit, in buffers cut from
lockstep's in the exact form: one CTA's worth of them (one large instance),
and several."""
import numpy as np
import pytest

from cases import contact_case
from spacelab_gb300 import BallGroup
from spacelab_gb300 import batch as B
from spacelab_gb300._lib import check

pytestmark = pytest.mark.gpu


def _run(counts, mode, refuse):
    cols = []
    for k, n in enumerate(counts):
        c = contact_case(n, 30 + k)
        col = B.Collision(n, 0, 0.0, 0.0, 0.6, 0.3, k)
        col.group = BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])
        col.dt, col.kin, col.kout = c["dt"], c["kin"], c["kout"]
        cols.append(col)
    run = B.BatchRun(cols, mode, steps=6, skip=2)
    run.set_shape(0, 128)
    assert run.shape()[2] > len(counts)  # lockstep
    if refuse:
        check(run.lib.sl_diag_batch_refuse_lockstep(run.h), "sl_diag_batch_refuse_lockstep")
    run.run(1, 3, do_init=True)
    run.run(4, 3, do_init=False)
    assert not run.status().any()
    blocks = run.shape()[2]
    out, energy = run.state(), run.energy()
    run.close()
    return blocks, out, energy


@pytest.mark.parametrize("mode", ["exact", "mixed_df"])
@pytest.mark.parametrize("counts", [[500, 40, 33], [130] * 9, [1]])
def test_the_per_cta_form_takes_over(mode, counts):
    _, want, e_want = _run(counts, mode, False)
    blocks, got, e_got = _run(counts, mode, True)
    assert 1 <= blocks <= len(counts)
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    scale = np.abs(e_want).max(axis=(1, 2), keepdims=True)
    assert (np.abs(e_got - e_want) <= 1e-10 * scale).all()
