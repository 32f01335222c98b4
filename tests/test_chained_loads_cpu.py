"""Chained kernels (launch_chained) start before the kernels in front have written
what they read, so those values may not come through the read-only path, which is
for memory that nobody writes during the kernel's life: no __ldg of a pointer that
went through chain_wait, or of the parts and partials handed on from one."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dplr_gb300", "csrc")


@pytest.mark.parametrize("name", ["apply.cu", "sweep.cuh", "fp64tile.cuh"])
def test_no_read_only_loads_of_what_a_kernel_in_front_writes(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    waited = {"parts", "parts_in", "partials"}
    for var, init in re.findall(r"\*\s*(\w+)\s*=\s*([^;]+);", text):
        if "chain_wait(" in init or set(re.findall(r"\w+", init)) & waited:
            waited.add(var)
    assert name == "fp64tile.cuh" or len(waited) > 3
    bad = [v for v in re.findall(r"__ldg\(\s*(\w+)", text) if v in waited]
    assert not bad, bad
