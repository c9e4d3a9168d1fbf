"""Which gradients of the log-likelihoods go to pcb_root_flows (host side)."""

import torch

from conftest import load_fixture
from helpers import build_fixture_circuit

from pyjuice_b200.model import tensorcircuit as mod


def test_gradients_that_the_kernel_reads(monkeypatch):
    """Plain FP32 gradients of the last batch's shape; wrapped ones, and every one where this torch
    cannot tell them apart, take the tensor operations."""
    pc = build_fixture_circuit("tiny", load_fixture("tiny"))
    pc.node_mars = torch.zeros([pc.num_nodes, 6])
    grad = torch.ones([6, pc.num_root_nodes])
    assert pc._takes_root_grad(grad)
    assert not pc._takes_root_grad(grad.double())
    assert not pc._takes_root_grad(grad[:5])
    seen = []
    torch.func.vmap(lambda g: (seen.append(pc._takes_root_grad(g)), g)[1])(torch.ones([2, 6, pc.num_root_nodes]))
    assert seen == [False]
    monkeypatch.setattr(torch._C, "_functorch", None)
    assert pc._takes_root_grad(grad)  # looked up once, when the module is loaded
    monkeypatch.setattr(mod, "_is_wrapped", None)
    assert not pc._takes_root_grad(grad)
