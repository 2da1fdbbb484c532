"""What a batch takes at its limits.  A batch too large for the lockstep form
makes none of its lists on the host (16 bytes per tile: 312 MB for one system
of 200,000 spheres, against a few MB)."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from cases import contact_case
from spacelab_gb300 import BallGroup
from spacelab_gb300 import batch as B

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

CREATE = """
import ctypes, resource, sys
sys.path.insert(0, {root!r})
from spacelab_gb300 import _lib, configs
lib = _lib.lib()
def make(counts, mode):
    h = ctypes.c_void_p()
    c = (ctypes.c_int * len(counts))(*counts)
    mat = configs.dust_material()
    _lib.check(lib.sl_batch_create(len(counts), c, ctypes.byref(mat), mode, 10, 10, ctypes.byref(h)), "sl_batch_create")
    return h
small = make([64], 0)
before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
large = make([200000], 0)
print(resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before)
lib.sl_batch_destroy(large)
lib.sl_batch_destroy(small)
"""


def test_a_large_system_makes_no_tile_lists():
    out = subprocess.run([sys.executable, "-c", CREATE.format(root=str(ROOT))], stdout=subprocess.PIPE, text=True,
                         timeout=300, check=True).stdout
    assert int(out) < 64 * 1024, out  # KB


def _collision(n, seed):
    c = contact_case(n, seed)
    col = B.Collision(n, 0, 0.0, 0.0, 0.6, 0.3, seed)
    col.group = BallGroup.from_arrays(c["pos"], c["vel"], c["w"], c["R"], c["m"], c["moi"])
    col.dt, col.kin, col.kout = c["dt"], c["kin"], c["kout"]
    return col


def _two_steps(cols, steps):
    run = B.BatchRun(cols, "mixed_df", steps=steps, skip=1)
    try:
        run.set_shape(0, 512)
        run.run(1, 2, do_init=True)
        return run.shape()[2], run.state()
    finally:
        run.close()


def test_the_required_memory_comes_first():
    """One system of 30,000 spheres: 0.68 GB for lockstep, as much for a CTA's
    partials.  4 GB are left free, and energy records are asked for that leave
    0.4 GB of them."""
    torch = pytest.importorskip("torch")
    cols = [_collision(30000, 3)]
    blocks, want = _two_steps(cols, 2)
    assert blocks > 1  # lockstep, with room
    left = 4 << 30
    hog = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        part = 24 * 938 * 938 * 32
        blocks, got = _two_steps(cols, (left - part - (400 << 20)) // 64)
    finally:
        del hog
        torch.cuda.empty_cache()
    assert blocks == 1  # an instance per CTA
    for k in want:
        assert np.array_equal(got[k], want[k]), k


def test_even_mixed_batches_hold_no_lockstep_memory():
    """4096 systems of 300 spheres: 0.56 GB of state and partials; lockstep,
    which they never take, would be 0.31 GB more."""
    torch = pytest.importorskip("torch")
    cols = [_collision(300, 3)] * 4096
    B.BatchRun(cols[:1], "mixed_df", steps=2, skip=1).close()  # the context's own memory
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    run = B.BatchRun(cols, "mixed_df", steps=2, skip=1)
    held = free - torch.cuda.mem_get_info()[0]
    run.set_shape(0, 64)
    assert run.shape()[2] > 152  # an instance per CTA, at the fewest threads too
    run.close()
    state = 4096 * 300 * (24 * 8 + 8 * 8 + 15 * 8 + 10 * 4 + 4)
    partials = 608 * 6 * 10 * 320 * 4
    assert held < state + partials + (100 << 20), held
