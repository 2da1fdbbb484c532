"""The double-float form's listed close pairs far from the origin: the search
adds the positions' lo parts there, so that pairs are right and no more of them
are listed.  Accelerations of a cluster without contacts against the exact form.

Bar: at 1e7 radii a displacement component is off by the two positions' 48 bits,
2^-47 1e7 = 7e-8 radii, and FP32's 1.2e-7; at gaps of 0.4 radii the force goes with
less than the gap's seventh power: 7 x 2e-7 / 0.4 = 3.5e-6, and some 2e-6 for
FP32's force arithmetic.  1e-5 of the norm.

The time per step may not grow with the distance: it did by 1.77 (every pair of
a tile was listed), now by 1.02."""
import time

import numpy as np
import pytest

from cases import RADIUS, contact_case, material
from spacelab_gb300 import BallGroup, GpuStep

pytestmark = pytest.mark.gpu


def _group(c, offset):
    return BallGroup.from_arrays(c["pos"] + offset * RADIUS, c["vel"], c["w"], c["R"], c["m"], c["moi"])


@pytest.mark.parametrize("spread", [0.0, 0.1])
@pytest.mark.parametrize("offset", [0.0, 1e5, 1e6, 1e7])
def test_forces(offset, spread):
    c = contact_case(333, 12, spacing=2.6, r_spread=spread)
    acc = {}
    for mode in ("exact", "mixed_df"):
        g = _group(c, offset)
        with GpuStep(g, material(), mode) as s:
            s.set_scalars(c["dt"], c["kin"], c["kout"])
            s.init_conditions()
            s.sim_looper(steps=2, skip=10)  # plain steps
            s.download()
        acc[mode] = g.acc
    assert np.linalg.norm(acc["mixed_df"] - acc["exact"]) <= 1e-5 * np.linalg.norm(acc["exact"])


def _step_time(offset):
    c = contact_case(1000, 3, spacing=2.1, vel_sigma=1e-3, w_sigma=1.0)
    with GpuStep(_group(c, offset), material(), "mixed_df") as s:
        s.set_scalars(c["dt"] * 1e-3, c["kin"], c["kout"])
        s.init_conditions()
        times = []
        for _ in range(8):
            t = time.perf_counter()
            s.sim_looper(steps=101, skip=100)
            times.append(time.perf_counter() - t)
    return min(times)


def test_time_does_not_grow_with_the_distance():
    assert _step_time(1e7) <= 1.3 * _step_time(0.0)
