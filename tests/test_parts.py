"""The FP64-accumulating mixed form's pair subtraction (csrc/sl_parts.cuh) on
the host.  An FP64 subtraction rounded once to FP32 is off by half a last
place; the three parts may add 2^-12 of one (their tail's own rounding is at
2^-22 of the result)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_differences_are_rounded_once(tmp_path):
    exe = tmp_path / "parts_check"
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-ffp-contract=off", "-Wall", "-Werror",
                    "-I", str(ROOT / "spacelab_gb300" / "csrc"), str(ROOT / "tests" / "parts_check.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), "2000000"], stdout=subprocess.PIPE, text=True, timeout=300, check=True).stdout
    rows = [line.split() for line in out.splitlines()]
    assert len(rows) == 5
    for distance, cases, worst in rows:
        assert float(worst) <= 0.5 + 2.0 ** -12, (distance, worst)
