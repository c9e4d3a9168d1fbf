"""The persistent tensor-memory contraction with many (tile, 128-sample slice) units per CTA: weight
slots taken over between slices and tiles, copied rows and accumulators across units."""

import pytest
import torch

import pyjuice_b200 as juice
from pyjuice_b200 import _native as nat
from pyjuice_b200.layer.layers import SumLayer
from pyjuice_b200.nodes.distributions import Categorical

pytestmark = pytest.mark.gpu


# one chunk, copied rows; fewer rows than 128 at an odd batch; 128 rows of four chunks (one weight slot
# beside the sums), 520 units
@pytest.mark.parametrize("regions,nodes,terms,bs,B", [(119, 128, 128, 32, 512), (80, 96, 112, 16, 260), (130, 128, 400, 16, 512)])
@pytest.mark.parametrize("form", [1, 2])
def test_many_units(regions, nodes, terms, bs, B, form, cuda_device, monkeypatch):
    nat.device_status()
    monkeypatch.setattr(SumLayer, "tmem", 0)
    monkeypatch.setattr(SumLayer, "bf16_form", form)
    with juice.set_block_size(bs):
        leaves = [juice.inputs(v, num_node_blocks=terms // bs, dist=Categorical(num_cats=2)) for v in range(2 * regions)]
        prods = [juice.multiply(leaves[2 * r], leaves[2 * r + 1]) for r in range(regions)]
        sums = [juice.summate(p, num_node_blocks=nodes // bs) for p in prods]
    juice.InputLayer(leaves, cum_nodes=bs)
    juice.ProdLayer(prods)
    layer = juice.SumLayer(sums, global_nid_start=bs, global_pid_start=bs ** 2, global_pfid_start=0,
                           node2tiednodes=dict()).to(cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(terms + B)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    w = torch.exp(-4.0 * rnd(regions, nodes, terms))
    w = w / w.sum(dim=2, keepdim=True)
    params = torch.cat([torch.zeros([bs ** 2], device=cuda_device),
                        w.reshape(regions, nodes // bs, bs, terms).permute(0, 1, 3, 2).reshape(-1)])
    em = -12.0 * rnd(regions, terms, B)
    ems = torch.cat([torch.full([bs, B], -float("inf"), device=cuda_device), em.reshape(-1, B)])
    nm = torch.zeros([bs + regions * nodes, B], device=cuda_device)
    layer(nm, ems, params, force_use_bf16=True)
    ref = torch.log(w.double() @ em.double().exp())
    # split products are within 3 * 2^-18, single ones within 2^-8 + 2^-16; 24 accumulations of 2^-23
    # and the approximations' 2^-21 stay below the rest of the bound
    tol = 2e-5 if form == 2 else 5e-3
    assert torch.all((nm[bs:].reshape(ref.shape).double() - ref).abs() <= tol + 4e-7 * ref.abs())
    nf = torch.softmax(3.0 * rnd(regions, nodes, B), dim=1)
    nms = torch.cat([torch.zeros([bs, B], device=cuda_device), ref.float().reshape(-1, B)])
    want = (w.double().transpose(1, 2) @ (nf.double() * torch.exp(-ref.float().double()))) * em.double().exp()
    for modify in (False, True):
        ef = torch.zeros_like(ems)
        layer.backward(torch.cat([torch.zeros([bs, B], device=cuda_device), nf.reshape(-1, B)]), ef, nms, ems, params,
                       None, allow_modify_flows=modify)
        # as above, and exponents of magnitude up to about 30 rounded three times
        assert torch.all((ef[bs:].reshape(want.shape).double() - want).abs() <= (tol + 1e-5) * want)
    assert nat.device_status() == 0
