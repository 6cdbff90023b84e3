"""What the kernels' sources have to keep for launches as programmatic dependents (no GPU needed).

A kernel may be resident while the one before it still writes: it waits for that one before anything else, and only
memory that no kernel writes may be read as constant (``__restrict__`` or ``__ldg``).
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gmxapi_gb300", "csrc")
# roots, spline moduli, inverse masses and the batch's table of systems are copied from the host before a launch;
# the others are arrays in shared memory
CONSTANT = {"roots", "bsp", "inv_mass", "sys"}
SHARED = {"nbfp_b", "nbfp_s", "lane_rec", "rec", "jx", "jt"}


def _sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as fh:
                yield name, re.sub(r"//[^\n]*|/\*.*?\*/", "", fh.read(), flags=re.S)


def test_only_constant_tables_are_read_as_constant():
    for name, text in _sources():
        for used in re.findall(r"__restrict__\s+(\w+)", text):
            assert used in CONSTANT | SHARED, (name, used)
        for used in re.findall(r"__ldg\(\s*&?(\w+)", text):
            assert used in CONSTANT, (name, used)


def test_kernels_wait_for_their_predecessor_first():
    kernels = 0
    for name, text in _sources():
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\([^{;]*\)\s*\{\s*([^;]*);", text):
            if m.group(1) == "k_fma_probe":  # launched on its own
                continue
            kernels += 1
            first = m.group(2).strip()
            if first.startswith("constexpr"):
                first = text[m.end():].split(";")[0].strip()
            assert first in ("pdl_begin()", "nbx::pdl_begin()"), (name, m.group(1), first)
    assert kernels >= 50
