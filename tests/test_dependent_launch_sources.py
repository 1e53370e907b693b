"""Kernels launched as programmatic dependents run while their predecessor still writes, so their sources use no read-only
loads: ``__ldg``, ``ld.global.nc`` and ``const __restrict__`` are defined only for data that nobody writes during the kernel."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "sparseflow_b200", "csrc")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
DEPENDENT = [f for f in SOURCES if "dependency_wait()" in _code(f)]


def test_every_dependent_launch_waits():
    launching = [f for f in SOURCES if re.search(r"launch_(dependent|kernel)\(", _code(f))]
    assert launching and set(launching) <= set(DEPENDENT)


@pytest.mark.parametrize("name", DEPENDENT)
def test_no_read_only_loads(name):
    assert not re.findall(r"__ldg|ld\.global(?:\.\w+)*\.nc|__restrict__", _code(name))
