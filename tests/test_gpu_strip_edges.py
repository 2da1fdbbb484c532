"""The exact form's tiles in strips (strip_from, csrc/sl_tile_exact.cuh) at the
edges of its rule on this device: the last system that is all strips, the first
with whole tiles, and the sizes around the first last round that is nearly full
without strips.  State and contacts against the oracle over three steps, one of
them a write step."""
import numpy as np
import pytest

from cases import OracleMaterial, contact_case, material
from spacelab_gb300 import BallGroup, GpuStep

pytestmark = pytest.mark.gpu


def _tiles(nb):
    return nb * (nb + 1) // 2


def _edges(num_sms):
    warps = 16 * num_sms
    nb = 1
    while 2 * _tiles(nb + 1) <= warps:
        nb += 1
    full = next(k for k in range(nb + 1, 10 * nb) if 10 * (_tiles(k) % warps) > 9 * warps)
    return {"all_strips": 32 * nb, "whole_tiles": 32 * nb + 1, "before_full": 32 * (full - 1), "full": 32 * full - 5}


@pytest.mark.parametrize("edge", ["all_strips", "whole_tiles", "before_full", "full"])
def test_edges_bit_identical(edge):
    torch = pytest.importorskip("torch")
    n = _edges(torch.cuda.get_device_properties(0).multi_processor_count)[edge]
    c = contact_case(n, 17)
    from oracle.oracle import CpuOracle
    o = CpuOracle(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"], OracleMaterial(), c["dt"], c["kin"], c["kout"])
    g = BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])
    with GpuStep(g, material(), "exact") as sim:
        sim.set_scalars(c["dt"], c["kin"], c["kout"])
        sim.init_conditions()
        o.init()
        for k in range(1, 4):
            e, eo = sim.sim_one_step(k == 2), o.step(k == 2)
            assert np.array_equal(sim.contacts(), o.contacts()), k
            if e is not None:
                assert abs(e.PE - eo[0]) <= 1e-10 * max(abs(eo[0]), abs(eo[1]))
        sim.download()
        st = o.state()
        for key in ("pos", "vel", "w", "acc", "aacc"):
            assert np.array_equal(getattr(sim.group, key), st[key]), key
