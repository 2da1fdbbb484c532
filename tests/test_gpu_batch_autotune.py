"""The autotuner takes lockstep, which is one form at any thread count, as one
candidate: it is timed once, and its time stands at each of its shapes."""
import pytest

from cases import contact_case
from spacelab_gb300 import BallGroup
from spacelab_gb300 import batch as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["exact", "mixed_df"])
def test_lockstep_is_timed_once(mode):
    cols = []
    for k, n in enumerate((600, 40, 33)):
        c = contact_case(n, k)
        col = B.Collision(n, 0, 0.0, 0.0, 0.6, 0.3, k)
        col.group = BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])
        col.dt, col.kin, col.kout = c["dt"], c["kin"], c["kout"]
        cols.append(col)
    run = B.BatchRun(cols, mode, steps=4, skip=2)
    times = run.autotune(2)["times_ms"]
    tiles = [v for k, v in times.items() if k.startswith("pairtiles")]
    assert len(times) == 12 and len(tiles) == 3 and len(set(tiles)) == 1 and tiles[0] > 0
    run.close()
