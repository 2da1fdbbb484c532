"""Materials and positions at the edges of the exact form's integer path
(csrc/sl_pair_fast.cuh), bit for bit against the CPU oracle, through every
entry point that runs the tiles: a negative Hamaker constant (repulsion), none
(no cohesion), spheres in a plane -- zeros of both signs -- and on a line, and a
cluster in which only some rows of a tile meet a zero component.
Block remainders, equal and unequal radii, write steps among them."""
import ctypes

import numpy as np
import pytest

from cases import MATERIAL, OracleMaterial, contact_case
from spacelab_gb300 import BallGroup, GpuStep, _lib
from spacelab_gb300 import batch as B
from spacelab_gb300._lib import Material

pytestmark = pytest.mark.gpu

STATE = ("pos", "vel", "w", "acc", "aacc")


def _repulsion(n, equal):
    return contact_case(n, 21, r_spread=0.0 if equal else 0.1, spacing=2.05), -MATERIAL["Ha"]


def _no_cohesion(n, equal):
    return contact_case(n, 22, r_spread=0.0 if equal else 0.1), 0.0


def _flat(c, axes):
    for k in axes:
        c["pos"][:, k] = np.where(np.arange(len(c["pos"])) % 3 == 0, -0.0, 0.0)
        c["vel"][:, k] = 0.0
    return c


def _plane(n, equal):
    c = contact_case(n, 23, r_spread=0.0 if equal else 0.1)
    side = int(np.ceil(n ** 0.5))
    g = np.stack(np.meshgrid(np.arange(side), np.arange(side), indexing="ij"), -1).reshape(-1, 2)[:n]
    c["pos"][:, :2] = (g + np.random.default_rng(4).normal(0.0, 0.01, (n, 2))) * 2.0 * c["R"].mean()
    c["w"][:, :2] = 0.0
    return _flat(c, [2]), MATERIAL["Ha"]


def _line(n, equal):
    c = contact_case(n, 24, r_spread=0.0 if equal else 0.1)
    c["pos"][:, 0] = (np.arange(n) - n / 2) * 2.0 * c["R"].mean()
    c["w"][:] = 0.0
    return _flat(c, [1, 2]), MATERIAL["Ha"]


def _some_rows(n, equal):
    c = contact_case(n, 25, r_spread=0.0 if equal else 0.1)
    c["pos"][n // 2::7, 1] = c["pos"][0, 1]
    return c, MATERIAL["Ha"]


CASES = {"repulsion": _repulsion, "no_cohesion": _no_cohesion, "plane": _plane, "line": _line, "some_rows": _some_rows}


def _oracle(c, Ha):
    from oracle.oracle import CpuOracle
    om = OracleMaterial()
    om.Ha = Ha
    return CpuOracle(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"], om, c["dt"], c["kin"], c["kout"])


def _group(c):
    return BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("equal", [False, True])
@pytest.mark.parametrize("n", [5, 33, 130, 1700])
def test_steps_bit_identical(name, equal, n):
    c, Ha = CASES[name](n, equal)
    o = _oracle(c, Ha)
    with GpuStep(_group(c), Material(**{**MATERIAL, "Ha": Ha}), "exact") as sim:
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
        for k in STATE:
            assert np.array_equal(getattr(sim.group, k).view(np.uint64), st[k].view(np.uint64)), k


@pytest.mark.parametrize("name", sorted(CASES))
def test_static_pass_bit_identical(name):
    torch = pytest.importorskip("torch")
    c, Ha = CASES[name](97, False)
    o = _oracle(c, Ha)
    o.init()
    dev = [torch.from_numpy(np.ascontiguousarray(c[k]).reshape(-1)).cuda() for k in ("pos", "vel", "w", "R", "m", "moi")]
    acc, aacc = (torch.zeros(3 * 97, dtype=torch.float64, device="cuda") for _ in range(2))
    mat = Material(**{**MATERIAL, "Ha": Ha})
    rc = _lib.lib().sl_forces_static(97, *[t.data_ptr() for t in dev], ctypes.byref(mat), c["kin"], c["kout"],
                                     acc.data_ptr(), aacc.data_ptr(), None, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert np.array_equal(acc.cpu().numpy().reshape(-1, 3), o.state()["acc"])


@pytest.mark.parametrize("name", sorted(CASES))
def test_batch_equals_single_steps(name, monkeypatch):
    """The batch's tiles against the per-instance oracle over three steps."""
    cs = [CASES[name](n, equal)[0] for n, equal in ((40, False), (97, True), (7, False))]
    Ha = CASES[name](7, False)[1]
    monkeypatch.setattr(B.configs, "dust_material", lambda: Material(**{**MATERIAL, "Ha": Ha}))
    cols = []
    for c in cs:
        col = B.Collision(len(c["R"]), 0, 0.0, 0.0, 0.6, MATERIAL["u_s"], 0)
        col.group, col.dt, col.kin, col.kout = _group(c), c["dt"], c["kin"], c["kout"]
        cols.append(col)
    run = B.BatchRun(cols, "exact", steps=3, skip=2)
    run.set_shape(0, 128)
    run.run(1, 3, do_init=True)
    got = run.state()
    run.close()
    off = 0
    for c in cs:
        o = _oracle(c, Ha)
        o.init()
        for k in range(1, 4):
            o.step(k == 2)
        for k in STATE:
            assert np.array_equal(got[k].reshape(-1, 3)[off:off + len(c["R"])], o.state()[k]), k
        off += len(c["R"])
