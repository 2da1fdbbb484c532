"""The exact pair force's integer path (spacelab_gb300/csrc/sl_pair_fast.cuh)
where a sign or a zero decides: on the host, results that it does not flag
against IEEE double operations."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def stats(tmp_path_factory):
    exe = tmp_path_factory.mktemp("pair") / "pair_signs_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wall", "-Werror", "-Wno-unknown-pragmas",
                    "-I", str(ROOT / "spacelab_gb300" / "csrc"), str(ROOT / "tests" / "pair_signs_check.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), "300000"], stdout=subprocess.PIPE, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
    return {line.split()[0]: [int(v) for v in line.split()[1:]] for line in out.stdout.splitlines()}


@pytest.mark.parametrize("case", ["repulsion", "plane", "line", "no_cohesion"])
def test_settled_results_are_ieee(stats, case):
    assert stats["mismatches"] == [0]
    cases, flagged = stats[case]
    assert cases >= 100_000 and flagged < 0.1 * cases
