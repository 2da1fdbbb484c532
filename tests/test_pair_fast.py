"""The unpacked integer arithmetic of the exact pair force
(spacelab_gb300/csrc/sl_pair_fast.cuh), checked on the host: the reciprocals'
errors against exact integers, and every result the header does not flag
against IEEE double operations.  The bounds are the ones its header derives
its rounding windows from."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_unflagged_results_are_ieee(tmp_path):
    exe = tmp_path / "pair_fast_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wall", "-Werror", "-Wno-unknown-pragmas",
                    "-I", str(ROOT / "spacelab_gb300" / "csrc"), str(ROOT / "tests" / "pair_fast_check.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), "2000000"], stdout=subprocess.PIPE, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
    stats = {line.split()[0]: [float(v) for v in line.split()[1:]] for line in out.stdout.splitlines()}
    assert stats["mismatches"] == [0.0], out.stdout
    # each path is exercised, and its flags are few
    for op in ("root", "quotient_root", "recip", "mass_recip", "product", "pairs"):
        cases, flagged = stats[op][:2]
        assert cases > 900_000 and flagged < 0.1 * cases, out.stdout
    # the bounds that the rounding windows allow for
    for op, lo, hi in (("recip_root", -2, 1), ("recip", -1, 2), ("mass_recip", -1, 0)):
        assert lo <= stats[op][2] and stats[op][3] <= hi, out.stdout
