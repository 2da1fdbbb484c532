"""The exact tile's two paths (csrc/sl_tile_exact.cuh) at the systems that
choose between them, bit for bit against the CPU oracle: constants outside
the integer path's range (no cohesion, very light spheres), equal radii with
unequal masses, lattices whose displacements have zero components, a tile
whose pairs are all in contact (a full list), and block remainders."""
import numpy as np
import pytest

from cases import MATERIAL, RADIUS, OracleMaterial, contact_case
from spacelab_gb300._lib import Material


def _lattice(n):
    c = contact_case(n, 3, r_spread=0.0)
    side = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    c["pos"] = g * 2.5 * RADIUS
    return c, {}


def _packed(n):  # every pair overlaps
    c = contact_case(n, 4)
    c["pos"] = c["pos"] / c["pos"].std() * 0.1 * RADIUS
    return c, {}


def _no_cohesion(n):
    return contact_case(n, 5), {"Ha": 0.0}


def _light(n):  # masses below 2^-200
    c = contact_case(n, 6)
    for k in ("m", "moi"):
        c[k] = c[k] * 2.0 ** -180
    for k in ("kin", "kout"):
        c[k] = c[k] * 2.0 ** -180
    return c, {"Ha": MATERIAL["Ha"] * 2.0 ** -180}


def _equal_radii(n):
    c = contact_case(n, 7, r_spread=0.0)
    c["m"] = c["m"] * np.linspace(0.5, 2.0, n)
    return c, {}


def _uniform(n):
    return contact_case(n, 8, r_spread=0.0, spacing=2.02), {}


@pytest.mark.gpu
@pytest.mark.parametrize("make,n", [(_lattice, 100), (_packed, 64), (_packed, 37), (_no_cohesion, 97), (_light, 65),
                                    (_equal_radii, 130), (_uniform, 31), (_uniform, 97), (_uniform, 400), (_packed, 250)])
def test_tile_paths_bit_identical(make, n):
    from oracle.oracle import CpuOracle
    from spacelab_gb300 import BallGroup, GpuStep
    c, mat = make(n)
    values = {**MATERIAL, **mat}
    om = OracleMaterial()
    for k, v in values.items():
        setattr(om, k, v)
    o = CpuOracle(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"], om, c["dt"], c["kin"], c["kout"])
    g = BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])
    with GpuStep(g, Material(**values), "exact") as sim:
        sim.set_scalars(c["dt"], c["kin"], c["kout"])
        sim.init_conditions()
        o.init()
        for k in range(1, 13):
            assert np.array_equal(sim.contacts(), o.contacts()), k
            e, eo = sim.sim_one_step(k % 4 == 0), o.step(k % 4 == 0)
            if e is not None:  # PE: mixed-sign terms, summed in another order
                assert abs(e.PE - eo[0]) <= 1e-10 * max(abs(eo[0]), abs(eo[1]))
        sim.download()
        st = o.state()
        for k in ("pos", "vel", "w", "acc", "aacc"):
            assert np.array_equal(getattr(sim.group, k), st[k]), k


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8, 9, 63, 1560, 1577, 2208, 2300])
def test_strips_bit_identical(n):
    """Tiles taken whole and in strips of 8 rows (pair_split): all of them (up
    to N=1560 on 152 SMs), the last ones (N=1577: the first system with whole
    tiles), none (N=2208), the last ones of a second round (N=2300); state and
    contacts against the oracle over three steps, one of them a write step."""
    from cases import material
    from oracle.oracle import CpuOracle
    from spacelab_gb300 import BallGroup, GpuStep
    c = contact_case(n, 9)
    o = CpuOracle(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"], OracleMaterial(), c["dt"], c["kin"], c["kout"])
    g = BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])
    with GpuStep(g, material(), "exact") as sim:
        sim.set_scalars(c["dt"], c["kin"], c["kout"])
        sim.init_conditions()
        o.init()
        for k in range(1, 4):
            assert np.array_equal(sim.contacts(), o.contacts()), k
            e, eo = sim.sim_one_step(k == 2), o.step(k == 2)
            if e is not None:
                assert abs(e.PE - eo[0]) <= 1e-10 * max(abs(eo[0]), abs(eo[1]))
                assert abs(e.KE - eo[1]) <= 1e-12 * abs(eo[1])
        sim.download()
        st = o.state()
        for key in ("pos", "vel", "w", "acc", "aacc"):
            assert np.array_equal(getattr(sim.group, key), st[key]), key


@pytest.mark.gpu
@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("n", [2, 33, 512, 513])
def test_write_step_potentials_apart_and_inline(n, overlap):
    """A write step's potentials in work items of their own (up to N=512 on
    152 SMs) and beside the forces (N=513), spheres 2.3 radii apart, so
    that PE is the near pairs' closed form and the far pairs' series alone.
    The closed form's own rounding, eps / w^2 of a far pair's w^3, is below
    1e-12 of the sum."""
    from cases import material
    from oracle.oracle import CpuOracle
    from spacelab_gb300 import BallGroup, GpuStep
    c = contact_case(n, 10, spacing=2.3)
    o = CpuOracle(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"], OracleMaterial(), c["dt"], c["kin"], c["kout"])
    g = BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])
    with GpuStep(g, material(), "exact") as sim:
        sim.set_overlap(overlap)
        sim.set_scalars(c["dt"], c["kin"], c["kout"])
        sim.init_conditions()
        o.init()
        for _ in range(2):
            e, eo = sim.sim_one_step(True), o.step(True)
            assert abs(e.PE - eo[0]) <= 1e-10 * abs(eo[0])
