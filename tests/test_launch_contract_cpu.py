"""Kernels launched as programmatic dependents start while the kernel before
them still writes their inputs, so they and the functions they call may not read
global memory by loads that require it to be unwritten for the kernel's whole life:
no __ldg, no const __restrict__ pointer parameters."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "molla_b200" / "csrc"
SHARED = {"vblock"}  # pointers to shared memory

FUNCTION = re.compile(r"(__global__|__device__)[^;{}()]*?(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(([^{};]*)\)\s*\{", re.S)


def functions(text):
    """name -> (is a kernel, parameters, body) of the functions of a CUDA source."""
    out = {}
    text = re.sub(r"//[^\n]*", "", text)
    for f in FUNCTION.finditer(text):
        depth, at = 1, f.end()
        while depth and at < len(text):
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        out[f.group(2)] = (f.group(1) == "__global__", f.group(3), text[f.end():at])
    return out


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu")))
def test_waiting_kernels_read_by_plain_loads(name):
    shared = functions((CSRC / "mpm_device.cuh").read_text())
    fns = {**shared, **functions((CSRC / name).read_text())}
    todo = [k for k, (kernel, _, body) in fns.items() if kernel and "wait_previous()" in body]
    if name in ("mpm_particles.cu", "mpm_kernels.cu", "mpm_sort.cu", "mpm_f64.cu"):
        assert todo, "the waiting kernels were not found"
    seen = set()
    while todo:
        k = todo.pop()
        if k in seen:
            continue
        seen.add(k)
        _, params, body = fns[k]
        assert "__ldg(" not in body, f"{k}: __ldg"
        for q in re.findall(r"const\s[^,]*?\*\s*__restrict__\s+(\w+)", params):
            assert q in SHARED, f"{k}: const __restrict__ {q}"
        assert not [q for q in re.findall(r"const\s[^;=(]*?\*\s*__restrict__\s+(\w+)\s*=", body) if q != "blk"], k
        todo += [c for c in fns if c not in seen and re.search(rf"\b{c}\s*(<[^;()]*>)?\(", body)]
