"""What a batch takes at its limits.  A batch too large for the lockstep form
makes none of its lists on the host (16 bytes per tile: 312 MB for one system
of 200,000 spheres, against a few MB)."""
import subprocess
import sys
from pathlib import Path

import pytest

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
