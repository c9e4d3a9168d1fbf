"""Tensor-memory columns are allocated so that no CTA can wait for good: an allocation waits while a
CTA holds the columns, which must not itself wait for this one. Read from the sources: a run could
only show it by hanging a GPU."""

import itertools
import os
import re

import pytest

from pyjuice_b200 import _native as nat

EARLY = "lse_tmem_kernel"              # allocates before its wait for the grid before
HELD_BACK = "sum_pflows_lanes_kernel"  # lets its successor start after its allocation


def _source(name):
    with open(os.path.join(nat.CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _kernels():
    for name in nat.SOURCES:
        for body in re.split(r"\b__global__\b", _source(name))[1:]:
            if "tmem_alloc(" in body:
                yield name, re.search(r"(\w+_kernel)\(", body).group(1), body


KERNELS = [pytest.param(*k, id=k[1]) for k in _kernels()]


def test_the_kernels_are_found():
    assert {k.id for k in KERNELS} >= {EARLY, HELD_BACK, "lse_tmem_persistent_kernel", "lse_tc05_kernel",
                                       "lse_tc05_ws_kernel", "sum_pflows_tc05_kernel"}


@pytest.mark.parametrize("name,kernel,body", KERNELS)
def test_order_of_wait_and_allocation(name, kernel, body):
    assert body.count("tmem_alloc(") == 1 and body.count("pdl_trigger()") == 1
    at = body.index("tmem_alloc(")
    if kernel == EARLY:
        return
    before = body[:at]
    assert "pdl_wait();" in before
    # by the warp that allocates: no barrier in between
    assert "__syncthreads" not in before[before.rindex("pdl_wait();"):]
    if kernel == HELD_BACK:
        assert re.search(r"tmem_alloc\([^;]*\);\s*pcb::pdl_trigger\(\);", body)


def test_what_shares_an_sm_fits_its_columns():
    """Columns and least shared memory (KB) of the CTAs that may be waiting for their allocation beside
    early ones, or that wait for others of their cluster: every set that fits an SM's 228 KB (1 KB more
    each) fits its 512 columns."""
    tmem = _source("lse_tmem.cu")
    kb = lambda text, name: int(re.search(name + r" = (\d+) \* 1024", text).group(1))
    pflows = int(re.search(r"static_assert\(smem >= (\d+) \* 1024", _source("sum_pflows_tc05.cu")).group(1))
    slices = int(re.search(r"static_assert\(smem >= (\d+) \* 1024", _source("lse_tc05.cu")).group(1))
    assert "std::max<size_t>(Smem(n_max, several, ksplit).total, kShared)" in tmem
    assert "std::max<size_t>(S.total, kPShared)" in tmem
    ctas = {"early": (256, kb(tmem, "kShared")), "persistent": (512, kb(tmem, "kPShared")), "pflows": (128, pflows),
            "slices": (128, slices)}
    for counts in itertools.product(range(4), repeat=len(ctas)):
        if counts[0] and sum(n * (k + 1) for n, (_, k) in zip(counts, ctas.values())) <= 228:
            assert sum(n * c for n, (c, _) in zip(counts, ctas.values())) <= 512, counts
