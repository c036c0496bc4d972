"""Registers and spills of kernels whose speed hangs on them, from the report
that the build leaves (the compiler's -Xptxas -v output)."""
import os
import re

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LOG = os.path.join(REPO, "_build", "ptxas_libgpg.log")
LIB = os.path.join(REPO, "gpu_testbed_poisson-gravity_b200", "lib", "libgpg.so")

# part of the mangled name, registers, bytes of spill stores and loads together
LIMITS = [
    ("14gravity_kernelIfLi1EE", 32, 0),     # eight CTAs of 256 threads per SM
    ("14gravity_kernelIfLi2EE", 32, 0),
    ("16sor_batch_kernelIfE", 128, 500),    # three and four CTAs per SM, bounded so
    ("16sor_batch_kernelIdE", 168, 500),
    ("17staged_sor_kernelIfLi2ELb1ELi2ELi2ELi2EE", 96, 50),
    ("17staged_sor_kernelIfLi3ELb1ELi2ELi2ELi1EE", 96, 0),
    ("17staged_sor_kernelIdLi3ELb1ELi2ELi2ELi1EE", 168, 50),
    ("17staged_sor_kernelIdLi4ELb0ELi2ELi2ELi1EE", 255, 0),
    ("10sor_kernelIdLi4ELi1ELb1ELi2ELi1EE", 128, 0),
]


@pytest.fixture(scope="module")
def report():
    if not os.path.exists(LOG) or (os.path.exists(LIB) and os.path.getmtime(LOG) + 600 < os.path.getmtime(LIB)):
        pytest.skip("no build report of this library")
    out, name, spill = {}, None, 0
    for line in open(LOG):
        m = re.search(r"Compiling entry function '(\S+)'", line)
        if m:
            name = m.group(1)
        m = re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", line)
        if m:
            spill = int(m.group(1)) + int(m.group(2))
        m = re.search(r"Used (\d+) registers", line)
        if m and name:
            out[name] = (int(m.group(1)), spill)
    return out


@pytest.mark.parametrize("kernel,registers,spill", LIMITS, ids=[k for k, _, _ in LIMITS])
def test_resources(report, kernel, registers, spill):
    found = [v for k, v in report.items() if kernel in k]
    assert len(found) == 1
    assert found[0][0] <= registers and found[0][1] <= spill
