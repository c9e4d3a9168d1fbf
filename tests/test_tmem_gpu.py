"""Contractions with the samples along the tensor-memory lanes (pcb_lse_contract_tmem) against
FP64: every launch form, at the edges of its tiles, chunks, slices and clusters."""

import pytest
import torch

import pyjuice_b200 as juice
from pyjuice_b200 import _native as nat
from pyjuice_b200.layer.layers import SumLayer
from pyjuice_b200.nodes.distributions import Categorical

pytestmark = pytest.mark.gpu


@pytest.fixture
def settings():
    names = ("tmem", "tc05_min_tiles", "bf16_form", "ratio_min_values")
    saved = {n: getattr(SumLayer, n) for n in names}
    yield
    for n, v in saved.items():
        setattr(SumLayer, n, v)


def _layer(regions, nodes, terms, bs, device):
    with juice.set_block_size(bs):
        leaves = [juice.inputs(v, num_node_blocks=terms // bs, dist=Categorical(num_cats=2)) for v in range(2 * regions)]
        prods = [juice.multiply(leaves[2 * r], leaves[2 * r + 1]) for r in range(regions)]
        sums = [juice.summate(p, num_node_blocks=nodes // bs) for p in prods]
    juice.InputLayer(leaves, cum_nodes=bs)
    juice.ProdLayer(prods)
    return juice.SumLayer(sums, global_nid_start=bs, global_pid_start=bs ** 2, global_pfid_start=0,
                          node2tiednodes=dict()).to(device)


# regions, nodes, terms, block, batch, ksplit (0: persistent), bf16 form
CASES = [(1, 16, 16, 16, 16, 1, 2), (3, 16, 128, 16, 129, 0, 2), (2, 144, 96, 16, 127, 1, 2), (2, 128, 128, 32, 128, 0, 1),
         (1, 64, 144, 16, 257, 1, 2), (2, 128, 256, 32, 130, 2, 2), (1, 96, 400, 16, 33, 3, 2), (1, 128, 640, 32, 200, 5, 2),
         (1, 48, 1040, 16, 100, 8, 2), (5, 128, 256, 32, 300, 0, 2), (3, 80, 656, 16, 140, 0, 2), (160, 32, 32, 32, 512, 0, 2),
         (40, 256, 256, 32, 260, 0, 2), (2, 128, 272, 16, 64, 8, 1)]


@pytest.mark.parametrize("regions,nodes,terms,bs,B,ksplit,form", CASES)
def test_contractions(regions, nodes, terms, bs, B, ksplit, form, cuda_device, settings):
    """Values and element flows (modified, unmodified through the kernel and through the ratio
    workspace), with samples that have no term above -inf and flows of zero."""
    SumLayer.tmem, SumLayer.tc05_min_tiles, SumLayer.bf16_form = ksplit, 1, form
    layer = _layer(regions, nodes, terms, bs, cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(nodes + terms + B)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    w = torch.exp(-4.0 * rnd(regions, nodes, terms))
    w = w / w.sum(dim=2, keepdim=True)
    params = torch.cat([torch.zeros([bs ** 2], device=cuda_device),
                        w.reshape(regions, nodes // bs, bs, terms).permute(0, 1, 3, 2).reshape(-1)])
    em = -12.0 * rnd(regions, terms, B)
    em[rnd(regions, terms, B) < 0.1] = -float("inf")
    em[0, :, 0] = -float("inf")  # a sample without any
    ems = torch.cat([torch.full([bs, B], -float("inf"), device=cuda_device), em.reshape(-1, B)])
    nm = torch.full([bs + regions * nodes, B], 5.0, device=cuda_device)
    layer(nm, ems, params, force_use_bf16=True)
    ref = torch.log(w.double() @ em.double().exp())
    got = nm[bs:].reshape(regions, nodes, B).double()
    # operand rounding: split products are within 3 * 2^-18, single ones within 2^-8 + 2^-16;
    # 24 accumulations of 2^-23 and the approximations' 2^-21 stay below the rest of the bound
    tol = 2e-5 if form == 2 else 5e-3
    assert torch.equal(torch.isinf(got), torch.isinf(ref))
    fin = torch.isfinite(ref)
    assert torch.all((got - ref)[fin].abs() <= tol + 4e-7 * ref[fin].abs())
    assert torch.all(nm[:bs] == 5.0)
    nm64 = ref.float().double()
    nms = torch.cat([torch.zeros([bs, B], device=cuda_device), ref.float().reshape(-1, B)])
    nf = torch.softmax(3.0 * rnd(regions, nodes, B), dim=1)
    nf[rnd(regions, nodes, B) < 0.1] = 0.0
    nfs = torch.cat([torch.zeros([bs, B], device=cuda_device), nf.reshape(-1, B)])
    ratio = torch.where(torch.isfinite(nm64), nf.double() * torch.exp(-nm64), 0.0)
    want = (w.double().transpose(1, 2) @ ratio) * em.double().exp()
    for modify, ratios in ((False, 1 << 62), (False, 0), (True, 0)):
        SumLayer.ratio_min_values = ratios
        flows = nfs.clone()
        ef = torch.full_like(ems, 9.0)
        layer.backward(flows, ef, nms, ems, params, None, allow_modify_flows=modify)
        assert modify or torch.equal(flows, nfs)
        out = ef[bs:].reshape(regions, terms, B).double()
        # as above, and exponents of magnitude up to about 30 rounded three times
        assert torch.all((out - want).abs() <= (tol + 1e-5) * want)
        assert torch.all(ef[:bs] == 9.0)
    assert nat.device_status() == 0


@pytest.mark.parametrize("regions,nodes,terms,bs,B", [(1, 64, 64, 32, 1), (2, 128, 128, 32, 129), (3, 80, 112, 16, 300),
                                                      (2, 128, 144, 16, 127), (1, 64, 400, 16, 260), (40, 128, 256, 32, 512)])
def test_fp32_form(regions, nodes, terms, bs, B, cuda_device, settings, monkeypatch):
    """The plain FP32 form on three-part operands: values and element flows against FP64."""
    from pyjuice_b200.layer import layers as mod
    SumLayer.tc05_min_tiles, SumLayer.ratio_min_values = 1, 0
    monkeypatch.setattr(mod, "_num_sms", lambda: 1)
    layer = _layer(regions, nodes, terms, bs, cuda_device)
    d = layer._desc(torch.device(cuda_device))
    assert layer._fw_f32(d, B) and all(layer._el_f32(eg, B) for eg in d["el_groups"])
    gen = torch.Generator(device=cuda_device).manual_seed(nodes + terms + B)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    w = torch.exp(-4.0 * rnd(regions, nodes, terms))
    w = w / w.sum(dim=2, keepdim=True)
    params = torch.cat([torch.zeros([bs ** 2], device=cuda_device),
                        w.reshape(regions, nodes // bs, bs, terms).permute(0, 1, 3, 2).reshape(-1)])
    em = -12.0 * rnd(regions, terms, B)
    em[rnd(regions, terms, B) < 0.1] = -float("inf")
    em[0, :, 0] = -float("inf")
    ems = torch.cat([torch.full([bs, B], -float("inf"), device=cuda_device), em.reshape(-1, B)])
    nm = torch.full([bs + regions * nodes, B], 5.0, device=cuda_device)
    layer(nm, ems, params, force_use_fp32=True)
    ref = torch.log(w.double() @ em.double().exp())
    got = nm[bs:].reshape(regions, nodes, B).double()
    assert torch.equal(torch.isinf(got), torch.isinf(ref))
    fin = torch.isfinite(ref)
    # exponents of magnitude up to 18 rounded twice (2 * 18 * 2^-24), the exponential's 2^-21, 10
    # truncations of 2^-23, the logarithm and the sum with the maximum 2 * 2^-24 of the value
    assert torch.all((got - ref)[fin].abs() <= 4e-6 + 2.0 ** -22 * ref[fin].abs())
    nms = torch.cat([torch.zeros([bs, B], device=cuda_device), ref.float().reshape(-1, B)])
    nf = torch.softmax(3.0 * rnd(regions, nodes, B), dim=1)
    nf[rnd(regions, nodes, B) < 0.1] = 0.0
    nfs = torch.cat([torch.zeros([bs, B], device=cuda_device), nf.reshape(-1, B)])
    nm64 = ref.float().double()
    ratio = torch.where(torch.isfinite(nm64), nf.double() * torch.exp(-nm64), 0.0)
    want = (w.double().transpose(1, 2) @ ratio) * em.double().exp()
    for modify in (False, True):
        ef = torch.full_like(ems, 9.0)
        layer.backward(nfs.clone(), ef, nms, ems, params, None, allow_modify_flows=modify, force_use_fp32=True)
        # as above with four roundings of exponents of magnitude up to 30
        assert torch.all((ef[bs:].reshape(regions, terms, B).double() - want).abs() <= 1.2e-5 * want)
        assert torch.all(ef[:bs] == 9.0)
    assert nat.device_status() == 0


@pytest.mark.parametrize("nodes,terms,bs,B,form", [(16, 16, 16, 1, 2), (128, 64, 32, 64, 2), (144, 80, 16, 65, 2), (256, 256, 32, 257, 2),
                                                   (48, 200, 8, 511, 2), (64, 128, 64, 130, 1)])
@pytest.mark.parametrize("children", [64, 128])
@pytest.mark.parametrize("modified", [False, True])
def test_lane_parameter_flows(nodes, terms, bs, B, form, children, modified, cuda_device):
    """pcb_sum_pflows_lanes: flows added to the slots, for tiles with fewer rows or children than
    a full one, the last samples of a chunk, zero flows and children without value."""
    layer = _layer(2, nodes, terms, bs, cuda_device)
    d = layer._desc(torch.device(cuda_device))
    gen = torch.Generator(device=cuda_device).manual_seed(nodes + B)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    w = rnd(2, nodes, terms) + 0.01
    pack = lambda x: x.reshape(2, nodes // bs, bs, terms).permute(0, 1, 3, 2).reshape(-1)
    params = torch.cat([torch.zeros([bs ** 2], device=cuda_device), pack(w)])
    em = -8.0 * rnd(2, terms, B)
    em[rnd(2, terms, B) < 0.1] = -float("inf")
    nm = -8.0 * rnd(2, nodes, B)
    nf = rnd(2, nodes, B)
    nf[rnd(2, nodes, B) < 0.1] = 0.0
    pad = lambda x, v: torch.cat([torch.full([bs, B], v, device=cuda_device), x.reshape(-1, B)])
    ems, nms = pad(em, -float("inf")), pad(nm, 0.0)
    flows = pad(nf.log() - nm, 0.0) if modified else pad(nf, 0.0)
    old = rnd(2 * nodes * terms)
    pf = old.clone()
    tiles = d["pf_tiles" if children == 64 else "pf_tiles128"]
    nat.call("pcb_sum_pflows_lanes", nat.ptr(flows), nat.ptr(nms), nat.ptr(ems), B, B, nat.ptr(params), nat.ptr(pf),
             nat.ptr(tiles), tiles.size(0), bs, nat.ptr(d["krow"]), nat.ptr(d["kw"]), nat.ptr(d["kpf"]),
             1 if modified else 0, 0, children, form, nat.stream())
    ratio = nf.double() * torch.exp(-nm.double())
    want = pack(w.double() * (ratio @ em.double().exp().transpose(1, 2)))
    # split operands: products within 3 * 2^-18; 36 accumulations truncated by 2^-23; exponents of
    # magnitude up to 24 rounded three times; the sum with the old value rounded once
    tol = (3.0 * 2.0 ** -18 if form == 2 else 2.0 ** -7) + 36 * 2.0 ** -23 + 1e-5
    assert torch.all((pf.double() - old.double() - want).abs() <= tol * want + 2.0 ** -23 * (old.double() + want))
    assert nat.device_status() == 0


@pytest.mark.parametrize("regions,nodes,terms,bs,B", [(1, 16, 16, 16, 1), (2, 128, 128, 32, 129), (3, 80, 272, 16, 260),
                                                      (2, 128, 656, 32, 131), (160, 32, 208, 16, 512)])
@pytest.mark.parametrize("form", [0, 1, 2])
def test_copied_rows(regions, nodes, terms, bs, B, form, cuda_device, settings, monkeypatch):
    """Persistent form: rows that come as 16-byte copies (aligned rows) and rows that are loaded by
    the threads (any other stride) go through the same arithmetic, to the bit."""
    from pyjuice_b200.layer import layers as mod
    SumLayer.tmem, SumLayer.tc05_min_tiles, SumLayer.ratio_min_values = 0, 1, 0
    monkeypatch.setattr(mod, "_num_sms", lambda: 1)
    if form:
        SumLayer.bf16_form = form
    layer = _layer(regions, nodes, terms, bs, cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(nodes + terms + B)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    params = torch.cat([torch.zeros([bs ** 2], device=cuda_device), rnd(regions * nodes * terms) / terms + 1e-4])
    em = -12.0 * rnd(bs + regions * terms, B)
    em[rnd(bs + regions * terms, B) < 0.1] = -float("inf")
    em[:, 0] = -float("inf")
    nf = torch.log(rnd(bs + regions * nodes, B)) + 6.0
    got = []
    for ld in (-(-B // 4) * 4 + 4, -(-B // 4) * 4 + 5):
        def at(t):
            m = torch.full([t.size(0), ld], float("nan"), device=cuda_device)  # nothing beyond B counts
            m[:, :B] = t
            return m[:, :B]
        nm, ef = at(torch.full([bs + regions * nodes, B], 5.0, device=cuda_device)), at(torch.full_like(em, 9.0))
        layer(nm, at(em), params, force_use_bf16=form != 0, force_use_fp32=form == 0)
        layer.backward(at(nf), ef, nm, at(em), params, None, allow_modify_flows=True, _flows_modified=True,
                       force_use_fp32=form == 0)
        got.append((nm.clone(), ef.clone()))
    (a, ea), (b, eb) = got
    assert not torch.isnan(a).any() and not torch.isnan(ea).any()
    assert torch.equal(a, b) and torch.equal(ea, eb)
    assert nat.device_status() == 0


def test_stored_choice_for_ratio_rows(cuda_device, settings, monkeypatch):
    """A stored choice of the TMA form for a layer's rewritten flows is not taken for the ratio
    workspace (which that form cannot read), nor one of the tensor-memory form when that is off."""
    from pyjuice_b200.autotune import TUNER
    SumLayer.tc05_min_tiles, SumLayer.ratio_min_values, SumLayer.tmem = 1, 0, None
    layer = _layer(2, 128, 128, 32, cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(3)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    params = torch.cat([torch.zeros([32 ** 2], device=cuda_device), rnd(2 * 128 * 128) / 128])
    ems, nms, nfs = -4.0 * rnd(32 + 256, 64), -rnd(32 + 256, 64), rnd(32 + 256, 64)

    def flows():
        ef = torch.zeros_like(ems)
        layer.backward(nfs.clone(), ef, nms, ems, params, None)
        return ef

    with monkeypatch.context() as m:
        m.setattr(TUNER, "choices", {})
        want = flows()
    for tmem, choice in ((None, ("ws", 64)), (False, ("tm", 9))):  # 9: no such form
        SumLayer.tmem = tmem
        nt = layer._desc(torch.device(cuda_device))["el_groups"][0]["tiles"].size(0)
        with monkeypatch.context() as m:
            m.setattr(TUNER, "choices", {"|".join(map(str, ("tc05", 1, 2, nt, 64))): choice})
            # split operands: the forms differ by their summation order and approximations
            assert torch.all((flows() - want).abs() <= 2e-5 * want.abs() + 1e-12)
    assert nat.device_status() == 0


@pytest.mark.parametrize("nodes,terms,bs,B", [(16, 144, 16, 16), (160, 160, 32, 33), (256, 256, 32, 64), (64, 320, 64, 512)])
def test_few_long_tiles(nodes, terms, bs, B, cuda_device):
    """One region of two to five 128-term chunks, default settings: split operands as in
    test_contractions, on whichever form the rules take."""
    layer = _layer(1, nodes, terms, bs, cuda_device)
    d = layer._desc(torch.device(cuda_device))
    assert layer._fw_long(d, 2) and layer._fw_long(d, 3) == (d["fw_ch"].size(0) >= 6)
    gen = torch.Generator(device=cuda_device).manual_seed(nodes + B)
    rnd = lambda *shape: torch.rand(shape, generator=gen, device=cuda_device)
    w = torch.exp(-4.0 * rnd(nodes, terms))
    w = w / w.sum(dim=1, keepdim=True)
    params = torch.cat([torch.zeros([bs ** 2], device=cuda_device),
                        w.reshape(nodes // bs, bs, terms).permute(0, 2, 1).reshape(-1)])
    em = -12.0 * rnd(terms, B)
    em[:, 0] = -float("inf")
    ems = torch.cat([torch.full([bs, B], -float("inf"), device=cuda_device), em])
    nm = torch.zeros([bs + nodes, B], device=cuda_device)
    layer(nm, ems, params, force_use_bf16=True)
    ref = torch.log(w.double() @ em.double().exp())
    got = nm[bs:].double()
    assert torch.equal(torch.isinf(got), torch.isinf(ref))
    fin = torch.isfinite(ref)
    assert torch.all((got - ref)[fin].abs() <= 2e-5 + 4e-7 * ref[fin].abs())
    nms = torch.cat([torch.zeros([bs, B], device=cuda_device), ref.float()])
    nf = torch.softmax(3.0 * rnd(nodes, B), dim=0)
    ef = torch.zeros_like(ems)
    layer.backward(torch.cat([torch.zeros([bs, B], device=cuda_device), nf]), ef, nms, ems, params, None)
    ratio = torch.where(fin, nf.double() * torch.exp(-ref), 0.0)
    want = (w.double().T @ ratio) * em.double().exp()
    assert torch.all((ef[bs:].double() - want).abs() <= 3e-5 * want)
