"""A handle given a new system: what sl_run captured for the old one -- the
mixed forms' length scale and far-pair threshold among it -- must not be used
for the new one.  Against a handle that never held the old system, bit for bit."""
import numpy as np
import pytest

from cases import contact_case, material
from spacelab_gb300 import BallGroup, GpuStep

pytestmark = pytest.mark.gpu


def _group(c, scale):
    return BallGroup.from_arrays(c["pos"] * scale, c["vel"] * scale, c["w"], c["R"] * scale, c["m"], c["moi"])


def _run(first, then, c, mode):
    g = first.copy()
    with GpuStep(g, material(), mode) as s:
        s.set_scalars(c["dt"], c["kin"], c["kout"])
        s.init_conditions()
        s.sim_looper(steps=21, skip=10)
        for k in ("pos", "vel", "w", "R", "m", "moi"):
            getattr(g, k)[:] = getattr(then, k)
        s.upload()
        s.init_conditions()
        s.sim_looper(steps=21, skip=10)
        s.download()
    return g


@pytest.mark.parametrize("mode", ["exact", "mixed", "mixed_df"])
@pytest.mark.parametrize("scale", [1.0, 64.0, 0.3])  # the same, larger and smaller radii
def test_interval_follows_the_upload(mode, scale):
    c = contact_case(100, 5)
    old, new = _group(c, 1.0), _group(c, scale)
    a, b = _run(old, new, c, mode), _run(new, new, c, mode)
    for k in ("pos", "vel", "w", "acc", "aacc"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
