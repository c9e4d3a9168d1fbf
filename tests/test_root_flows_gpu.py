"""Root flows in one launch: against FP64 over strides, roots and batch sizes, and the gradient
hook's route against the one through ``ll_weights``."""

import pytest
import torch

import pyjuice_b200 as juice
from pyjuice_b200 import _native as nat
from pyjuice_b200.model.tensorcircuit import TensorCircuit
from pyjuice_b200.nodes.distributions import Categorical

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("roots,B", [(1, 1), (1, 33), (3, 1000), (1, 8193), (2, 32768)])
@pytest.mark.parametrize("layout", ["rows", "columns", "expanded"])
@pytest.mark.parametrize("logspace", [False, True])
def test_root_flows(roots, B, layout, logspace, cuda_device):
    """The FP32 result of a rounded sum, one division and one product: three roundings, 4 x 2^-24
    of the value with their products (log: that much absolutely, and two units in the last place)."""
    gen = torch.Generator(device=cuda_device).manual_seed(B)
    g = torch.rand([B, roots], generator=gen, device=cuda_device) + 0.1
    if layout == "columns":
        g = g.T.contiguous().T
    elif layout == "expanded":
        g = g[:1, :1].expand(B, roots)
    ld = B + 3
    nf = torch.full([roots + 2, ld], 7.0, device=cuda_device)
    cum = torch.full([], 2.5, dtype=torch.float64, device=cuda_device)
    nat.call("pcb_root_flows", nat.ptr(g), g.stride(1), g.stride(0), roots, B, nat.ptr(nf[1]), ld, int(logspace),
             nat.ptr(cum), nat.stream())
    w = g.T.double() / g.double().sum() * B
    got = nf[1:1 + roots, :B].double()
    if logspace:
        assert torch.all((got - w.log()).abs() <= 4 * 2.0 ** -24 + 2.0 ** -22 * w.log().abs())
    else:
        assert torch.all((got - w).abs() <= 4 * 2.0 ** -24 * w)
    assert abs(cum.item() - 2.5 - B) <= 4 * 2.0 ** -24 * B
    nf[1:1 + roots, :B] = 7.0
    assert torch.all(nf == 7.0)


@pytest.mark.parametrize("form", ["mean", "sum", "weighted", "transposed", "partial"])
def test_hook_routes_agree(form, cuda_device, monkeypatch):
    """Both routes of the gradient hook: root flows within the roundings of FP32 sums of 130 terms,
    flows and the total of the root flows accordingly."""
    with juice.set_block_size(2):
        leaves = [juice.inputs(v, num_node_blocks=2, dist=Categorical(num_cats=3)) for v in range(2)]
        root = juice.summate(juice.multiply(*leaves), num_node_blocks=1, block_size=1)
    pc = juice.compile(root).to(cuda_device)
    x = torch.randint(0, 3, [130, 2], generator=torch.Generator().manual_seed(1)).to(cuda_device)
    scale = torch.linspace(0.5, 2.0, 130, device=cuda_device)[:, None]
    got = []
    for fused in (True, False):
        calls = []
        takes = TensorCircuit._takes_root_grad
        with monkeypatch.context() as m:
            m.setattr(TensorCircuit, "_takes_root_grad",
                      lambda self, g: calls.append(takes(self, g)) or (calls[-1] and fused))
            pc._cum_flow_dev = None
            pc.init_param_flows(flows_memory=0.0)
            lls = pc(x, force_use_fp32=True)
            if form == "weighted":
                (lls * scale).sum().backward()
            elif form == "transposed":
                lls.backward(gradient=scale.T.contiguous().T.expand(130, lls.size(1)))
            elif form == "partial":
                lls[::3].mean().backward()
            else:
                getattr(lls, form)().backward()
        assert calls == [True]
        r0, r1 = pc._root_node_range
        got.append((pc.node_flows[r0:r1].clone(), pc.param_flows.clone(), pc._cum_flow))
    (a, pa, ca), (b, pb, cb) = got
    tol = 130 * 2.0 ** -24
    assert torch.all((a - b).abs() <= tol * b.abs())
    assert torch.all((pa - pb).abs() <= 2 * tol * pb.abs())
    assert abs(ca - cb) <= tol * cb
