"""Kernels launched as programmatic dependents (csrc/sl_pdl.cuh) are resident
while their predecessors write what they read, so no non-coherent load may
stand in them or in a function that they call: neither __ldg nor a
__restrict__ pointer.  Read from the sources: on a GPU a stale line would show
only now and then."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "spacelab_gb300" / "csrc"


def _strip_comments(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _functions(text):
    """(name, text from the line of the definition to its closing brace)"""
    out = []
    for m in re.finditer(r"^[^\n;#{}]*(?:__global__|__device__)[^;{}]*\{", text, flags=re.M):
        head = re.sub(r"__launch_bounds__\s*\([^{]*?\)\s+(?=\w+\s*\()", " ", m.group(0))
        name = re.search(r"([A-Za-z_]\w*)\s*\(", head)
        depth, end = 1, m.end()
        while depth and end < len(text):
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        out.append((name.group(1) if name else "", text[m.start():end]))
    return out


SOURCES = {p.name: _strip_comments(p.read_text()) for p in sorted(CSRC.glob("*.cu*")) if p.name != "sl_pdl.cuh"}
BODIES = {}
for _text in SOURCES.values():
    for _name, _body in _functions(_text):
        BODIES.setdefault(_name, []).append(_body)
WAITING = sorted(n for n, bodies in BODIES.items() if any("pdl_wait()" in b for b in bodies))


def _reached(name):
    seen, todo = set(), [name]
    while todo:
        n = todo.pop()
        if n in seen:
            continue
        seen.add(n)
        for body in BODIES[n]:
            todo += [c for c in set(re.findall(r"\b([A-Za-z_]\w*)\s*(?:<[^;(){}]*>)?\s*\(", body)) if c in BODIES]
    return seen


def test_the_waiting_kernels_are_found():
    assert {"drift_kernel", "pair_tile_kernel", "energy_partial_kernel", "gemm_nt_tc_kernel", "mse_grad_kernel",
            "adam_kernel", "mixed64_pair_kernel", "mixed_pair_listed_kernel"} <= set(WAITING)
    assert "bias_grad" in _reached("gemm_nt_tc_kernel")


@pytest.mark.parametrize("kernel", WAITING)
def test_no_non_coherent_loads(kernel):
    for name in sorted(_reached(kernel)):
        for body in BODIES[name]:
            assert "__ldg" not in body and "ld.global.nc" not in body, (kernel, name)
            assert "__restrict__" not in body, (kernel, name)
