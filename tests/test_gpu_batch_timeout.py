"""A lockstep run whose wait between two phases runs out: it returns
SL_ERR_TIMEOUT, and a batch that is given a new state afterwards behaves like
a new one, bit for bit.  The barrier after the first pairs phase gives up, where
the contacts' torques are marked and not yet added; the new state has none.  The
row blocks are spread over several CTAs, as the last one to arrive goes on."""
import numpy as np
import pytest

from cases import contact_case
from spacelab_gb300 import BallGroup, _lib
from spacelab_gb300 import batch as B
from spacelab_gb300._lib import check, dptr

pytestmark = pytest.mark.gpu


def _cols(spacing):
    cols = []
    for k, n in enumerate((1500, 700, 33)):
        c = contact_case(n, 60 + k, spacing=spacing, vel_sigma=1.0, w_sigma=1e3)
        col = B.Collision(n, 0, 0.0, 0.0, 0.6, 0.3, k)
        col.group = BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])
        col.dt, col.kin, col.kout = c["dt"], c["kin"], c["kout"]
        cols.append(col)
    return cols


def _upload(run, cols):
    cat = lambda k: np.ascontiguousarray(np.concatenate([getattr(c.group, k) for c in cols])).reshape(-1)  # noqa: E731
    par = [np.array([getattr(c, k) for c in cols], dtype=np.float64) for k in ("dt", "kin", "kout", "mu")]
    check(run.lib.sl_batch_upload(run.h, *[dptr(a) for a in (*map(cat, ("pos", "vel", "w", "R", "m", "moi")), *par)]),
          "sl_batch_upload")


def _four_steps(run):
    run.run(1, 4, do_init=True)
    out = {**run.state(), "energy": run.energy()}
    run.close()
    return out


@pytest.mark.parametrize("mode", ["mixed_df", "exact"])
def test_a_new_state_after_a_timeout(mode):
    touching, apart = _cols(1.9), _cols(3.0)
    run = B.BatchRun(touching, mode, steps=4, skip=2)
    run.set_shape(0, 128)
    check(run.lib.sl_diag_batch_give_up(run.h, 2), "sl_diag_batch_give_up")
    with pytest.raises(_lib.SpaceLabError) as err:
        run.run(1, 4, do_init=True)
    assert err.value.code == _lib.SL_ERR_TIMEOUT
    check(run.lib.sl_diag_batch_give_up(run.h, 0), "sl_diag_batch_give_up")
    _upload(run, apart)
    got = _four_steps(run)
    fresh = B.BatchRun(apart, mode, steps=4, skip=2)
    fresh.set_shape(0, 128)
    want = _four_steps(fresh)
    assert not want["aacc"].any()  # no contacts, so no torques
    for k in want:
        assert np.array_equal(got[k], want[k]), k
