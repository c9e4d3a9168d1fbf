"""The forms that the row kernels' launch rules choose between give the same values: sizes on both
sides of each rule, and either form where a call names it."""

import pytest
import torch

import pyjuice_b200 as juice
from pyjuice_b200 import _native as nat
from pyjuice_b200.nodes.distributions import Categorical

pytestmark = pytest.mark.gpu


# few and many rows, rows with 16-byte accesses (four at a time from 227,328 threads on) and without
@pytest.mark.parametrize("rows,B", [(1, 1), (3, 33), (64, 64), (1023, 200), (6000, 512), (7104, 512), (7107, 516), (7107, 514)])
def test_flow_ratios(rows, B, cuda_device):
    gen = torch.Generator(device=cuda_device).manual_seed(rows + B)
    nf = torch.rand([rows + 2, B], generator=gen, device=cuda_device)
    nm = -4.0 * torch.rand([rows + 2, B], generator=gen, device=cuda_device)
    nf[torch.rand([rows + 2, B], generator=gen, device=cuda_device) < 0.1] = 0.0
    nm[0], nm[-1] = -float("inf"), -float("inf")
    ref = torch.where(torch.isinf(nm), -float("inf"), nf.double().log() - nm.double())
    out = torch.full([rows + 1, B], 7.0, device=cuda_device)
    nat.call("pcb_flow_ratios", nat.ptr(nf), nat.ptr(nm), nat.ptr(out), B, B, 0, rows, nat.stream())
    flows = nf.clone()
    nat.call("pcb_modify_flows", nat.ptr(flows), nat.ptr(nm), B, B, 1, rows + 2, nat.stream())
    for got, want in ((out[:rows], ref[:rows]), (flows[1:], ref[1:])):
        assert torch.equal(torch.isinf(got), torch.isinf(want))
        fin = torch.isfinite(want)
        # logf within 1 ulp of a magnitude up to 17, the difference rounded once
        assert torch.all((got.double() - want)[fin].abs() <= 2.0 ** -19 + 2.0 ** -24 * want[fin].abs())
    assert torch.all(out[rows] == 7.0) and torch.equal(flows[0], nf[0])
