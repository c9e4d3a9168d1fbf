"""Plain FP32 contractions of large layers (force_use_fp32): the accuracy of FP32 arithmetic over
its whole range, whichever kernel the layer's size selects."""

import pytest
import torch

import pyjuice_b200 as juice
from pyjuice_b200 import _native as nat
from pyjuice_b200.nodes.distributions import Categorical

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def clear_status():
    nat.device_status()


def _layer(regions, nodes, terms, bs, device):
    with juice.set_block_size(bs):
        leaves = [juice.inputs(v, num_node_blocks=terms // bs, dist=Categorical(num_cats=2)) for v in range(2 * regions)]
        prods = [juice.multiply(leaves[2 * r], leaves[2 * r + 1]) for r in range(regions)]
        sums = [juice.summate(p, num_node_blocks=nodes // bs) for p in prods]
    juice.InputLayer(leaves, cum_nodes=bs)
    juice.ProdLayer(prods)
    return juice.SumLayer(sums, global_nid_start=bs, global_pid_start=bs ** 2, global_pfid_start=0,
                          node2tiednodes=dict()).to(device)


def _params(w, bs, device):
    regions, nodes, terms = w.shape
    return torch.cat([torch.zeros([bs ** 2], device=device),
                      w.reshape(regions, nodes // bs, bs, terms).permute(0, 1, 3, 2).reshape(-1)])


@pytest.mark.parametrize("regions,nodes,terms,bs,B", [(119, 128, 128, 32, 512), (40, 96, 96, 32, 512), (60, 64, 272, 16, 260)])
def test_mean_error(regions, nodes, terms, bs, B, cuda_device):
    """Sums rounded to nearest have no direction: over some 10^6 values the errors cancel down to
    the lean of the exponential's and logarithm's approximations. 2^-24, half a unit in the last
    place of 1, is the most that a mean of relative errors of rounded sums can be; a truncating
    accumulator leaves several times that."""
    layer = _layer(regions, nodes, terms, bs, cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(terms + B)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    w = torch.exp(-4.0 * rnd(regions, nodes, terms))
    w = w / w.sum(dim=2, keepdim=True)
    # maxima at zero and logarithms of magnitude below 8, so that their own rounding stays small
    em = -12.0 * rnd(regions, terms, B)
    em = em - em.amax(dim=1, keepdim=True)
    ems = torch.cat([torch.full([bs, B], -float("inf"), device=cuda_device), em.reshape(-1, B)])
    nm = torch.zeros([bs + regions * nodes, B], device=cuda_device)
    layer(nm, ems, _params(w, bs, cuda_device), force_use_fp32=True)
    err = nm[bs:].reshape(regions, nodes, B).double() - torch.log(w.double() @ em.double().exp())
    assert err.mean().abs().item() <= 2.0 ** -24
    assert nat.device_status() == 0


@pytest.mark.parametrize("regions,nodes,terms,bs,B", [(40, 128, 128, 32, 512), (60, 64, 272, 16, 260)])
@pytest.mark.parametrize("gap", [60.0, 72.0, 80.0, 84.0, 95.0])
def test_zero_weight_on_the_largest_terms(regions, nodes, terms, bs, B, gap, cuda_device):
    """A node whose largest terms have weight zero (zeros kept by EM, tables with zeros) is the sum
    of terms ``gap`` nats below the tile's maximum."""
    layer = _layer(regions, nodes, terms, bs, cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(terms + B)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    w = rnd(regions, nodes, terms) + 0.1
    w[:, :, :terms // 2] = 0.0
    w = w / w.sum(dim=2, keepdim=True)
    em = -rnd(regions, terms, B)
    em[:, 0] = 0.0
    em[:, terms // 2:] -= gap - 0.5
    ems = torch.cat([torch.full([bs, B], -float("inf"), device=cuda_device), em.reshape(-1, B)])
    nm = torch.zeros([bs + regions * nodes, B], device=cuda_device)
    layer(nm, ems, _params(w, bs, cuda_device), force_use_fp32=True)
    err = nm[bs:].reshape(regions, nodes, B).double() - torch.log(w.double() @ em.double().exp())
    # exponents of magnitude up to 86 (138 in base 2) rounded twice, 2 * 138 ln 2 * 2^-24; up to 136
    # additions of 2^-24; the exponential's 2^-21, the logarithm and the sum with the maximum, 2 *
    # 2^-24 of 87. Products below the smallest normal number (84 nats and a weight of 2^-9) keep
    # 2^-150 of 2^-128.5 each. Subnormal terms (95 nats: 2^-139.2 times weights of 2^-4.9 to 2^-11)
    # are whole multiples of 2^-149: up to half of one off, per term, of a sum of 2^-138.
    tol = 4e-5 if gap < 90 else 0.1
    assert torch.all(err.abs() <= tol)
    assert nat.device_status() == 0


@pytest.mark.parametrize("regions,nodes,terms,bs,B", [(119, 128, 128, 32, 512), (80, 96, 112, 16, 260), (60, 64, 272, 16, 260)])
def test_three_part_form(regions, nodes, terms, bs, B, cuda_device, monkeypatch):
    """The form that ``SumLayer.fp32_parts`` asks for, with many units per SM: values and element
    flows within its bound (terms within 12 nats of the largest)."""
    from pyjuice_b200.layer.layers import SumLayer
    monkeypatch.setattr(SumLayer, "fp32_parts", True)
    layer = _layer(regions, nodes, terms, bs, cuda_device)
    d = layer._desc(cuda_device)
    assert layer._fw_parts(d, 0, B) and all(layer._el_parts(eg, 0, B) for eg in d["el_groups"])
    gen = torch.Generator(device=cuda_device).manual_seed(terms + B)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    w = torch.exp(-4.0 * rnd(regions, nodes, terms))
    w = w / w.sum(dim=2, keepdim=True)
    params = _params(w, bs, cuda_device)
    em = -12.0 * rnd(regions, terms, B)
    ems = torch.cat([torch.full([bs, B], -float("inf"), device=cuda_device), em.reshape(-1, B)])
    nm = torch.zeros([bs + regions * nodes, B], device=cuda_device)
    layer(nm, ems, params, force_use_fp32=True)
    ref = torch.log(w.double() @ em.double().exp())
    # exponents of magnitude up to 18 rounded twice (2 * 18 * 2^-24), the exponential's 2^-21, 10
    # truncations of 2^-23, the logarithm and the sum with the maximum 2 * 2^-24 of the value
    assert torch.all((nm[bs:].reshape(ref.shape).double() - ref).abs() <= 4e-6 + 2.0 ** -22 * ref.abs())
    nms = torch.cat([torch.zeros([bs, B], device=cuda_device), ref.float().reshape(-1, B)])
    nf = torch.softmax(3.0 * rnd(regions, nodes, B), dim=1)
    ef = torch.zeros_like(ems)
    layer.backward(torch.cat([torch.zeros([bs, B], device=cuda_device), nf.reshape(-1, B)]), ef, nms, ems, params,
                   None, allow_modify_flows=True, force_use_fp32=True)
    want = (w.double().transpose(1, 2) @ (nf.double() * torch.exp(-ref.float().double()))) * em.double().exp()
    # as above with four roundings of exponents of magnitude up to 30
    assert torch.all((ef[bs:].reshape(want.shape).double() - want).abs() <= 1.2e-5 * want)
    assert nat.device_status() == 0
