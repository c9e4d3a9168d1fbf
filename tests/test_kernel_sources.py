"""Rules that the kernel sources keep and no run can show without hanging a GPU."""

import os
import re

import pytest

from pyjuice_b200 import _native as nat


def _kernels():
    for name in nat.SOURCES:
        with open(os.path.join(nat.CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for body in re.split(r"\b__global__\b", text)[1:]:
            if "tmem_alloc(" in body:
                yield name, re.search(r"(\w+)\(", re.sub(r"__launch_bounds__\([^{]*?\)\n", "", body)).group(1), body


def test_there_are_such_kernels():
    assert len(list(_kernels())) >= 6


@pytest.mark.parametrize("name,kernel,body", [pytest.param(*k, id=f"{k[0]}:{k[1]}") for k in _kernels()])
def test_dependents_start_after_the_tensor_memory_is_allocated(name, kernel, body):
    """A dependent CTA may hold tensor-memory columns while it waits for this grid, so this grid's
    CTAs have theirs before they let it start: the one trigger is the next statement of the warp
    that allocates."""
    assert "pdl_begin()" not in body and body.count("pdl_trigger()") == 1
    assert re.search(r"if \(warp == \w+\) \{\s*tmem_alloc\([^;]*\);\s*pcb::pdl_trigger\(\);", body)
