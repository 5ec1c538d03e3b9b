"""The rule of a chained (programmatic) launch, read from the kernels' source: its blocks may be resident
while the kernel before it still writes, so the kernel waits for that one, and none of its pointers is
declared read-only for its whole life."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gregpackagescpp_b200", "csrc")


def _kernels():
    """(file, name, parameters, body) of every __global__ function."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            text = f.read()
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(([^)]*)\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield os.path.basename(path), m.group(1), m.group(2), text[m.end():end]


def test_no_restrict_in_waiting_kernels():
    waiting = [k for k in _kernels() if "cudaGridDependencySynchronize" in k[3]]
    assert len(waiting) >= 16, [k[1] for k in waiting]
    assert [k[:2] for k in waiting if "__restrict__" in k[2] or "__ldg(" in k[3] or "ld.global.nc" in k[3]] == []


def test_chained_kernels_wait():
    """Every kernel named in a launch_chained call waits for the one before it."""
    kernels = {k[1]: k[3] for k in _kernels()}
    named = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            for call in re.findall(r"launch_chained\(([^;]*);", f.read()):
                named |= set(re.findall(r"\b(\w+_kernel)\b", call))
    assert len(named) >= 12, named
    assert [k for k in sorted(named) if "cudaGridDependencySynchronize()" not in kernels[k]] == []
