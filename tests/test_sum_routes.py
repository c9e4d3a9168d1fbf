"""Which entry points a sum layer calls, and which calls it refuses before any launch: the host
side alone, with the launches recorded instead of made."""

import pytest
import torch

import pyjuice_b200 as juice
from pyjuice_b200 import _native as nat
from pyjuice_b200.layer import layers as mod
from pyjuice_b200.layer.layers import SumLayer
from pyjuice_b200.nodes.distributions import Categorical


@pytest.fixture
def calls(monkeypatch):
    """The entry points called, in order."""
    names = []
    monkeypatch.setattr(nat, "call", lambda name, *args: names.append(name))
    monkeypatch.setattr(nat, "stream", lambda: None)
    monkeypatch.setattr(nat, "ptr", lambda t: None)
    monkeypatch.setattr(mod, "_num_sms", lambda: 148)
    return names


def _layer(regions, nodes, terms, bs):
    with juice.set_block_size(bs):
        leaves = [juice.inputs(v, num_node_blocks=terms // bs, dist=Categorical(num_cats=2)) for v in range(2 * regions)]
        prods = [juice.multiply(leaves[2 * r], leaves[2 * r + 1]) for r in range(regions)]
        sums = [juice.summate(p, num_node_blocks=nodes // bs) for p in prods]
    juice.InputLayer(leaves, cum_nodes=bs)
    juice.ProdLayer(prods)
    return juice.SumLayer(sums, global_nid_start=bs, global_pid_start=bs ** 2, global_pfid_start=0, node2tiednodes=dict())


def _buffers(layer, B, ld=None):
    """Node values, node flows, element values, element flows: B columns of rows ``ld`` apart."""
    rows = layer._layer_nid_range[1], max(int(c.max()) for c in layer.partitioned_chids) + 128
    return [torch.zeros([n, ld or B])[:, :B] for n in (rows[0], rows[0], rows[1], rows[1])]


@pytest.mark.parametrize("nodes,terms,B", [(128, 128, 512), (64, 272, 260), (96, 96, 8)])
def test_plain_fp32_arithmetic(nodes, terms, B, calls):
    """force_use_fp32, and batches below 16, take the FP32 kernels whatever the layer's size."""
    layer = _layer(100, nodes, terms, 32 if terms % 32 == 0 else 16)
    nm, nf, em, ef = _buffers(layer, B)
    params = torch.zeros([1])
    layer(nm, em, params, force_use_fp32=B >= 16)
    for modify in (False, True):
        layer.backward(nf, ef, nm, em, params, None, allow_modify_flows=modify, force_use_fp32=B >= 16)
    assert set(calls) <= {"pcb_lse_contract", "pcb_lse_contract_short", "pcb_modify_flows"}


@pytest.mark.parametrize("which", [1, 2, 3])
@pytest.mark.parametrize("cut", [slice(8, None), slice(None, -8)])
def test_backward_refuses_other_widths(which, cut, calls):
    """Flows or values with other columns than the node values (same row stride) are refused before
    the first launch, where there are too few of them and, once parameter flows are summed over
    them, also where there are more; without parameter flows wider buffers serve as before."""
    layer = _layer(4, 64, 64, 32)
    bufs = _buffers(layer, 64, ld=72)
    narrow = list(bufs)
    narrow[which] = narrow[which][:, cut]
    order = lambda b: (b[1], b[3], b[0], b[2], torch.zeros([1]))
    pf = torch.zeros([1])
    for flows in (None, pf):
        with pytest.raises(ValueError):
            layer.backward(*order(narrow), flows)
    wide = [b if i == which else b[:, cut] for i, b in enumerate(bufs)]
    if which != 3:
        with pytest.raises(ValueError):
            layer.backward(*order(wide), pf)
    assert calls == []
    layer.backward(*order(wide), None)
    assert calls != []


@pytest.mark.parametrize("nodes,terms", [(160, 160), (256, 256), (64, 320), (1024, 1024)])
def test_without_the_tensor_memory_form(nodes, terms, calls, monkeypatch):
    """``SumLayer.tmem = False`` brings back the kernels that long tiles had without it: mma.sync
    below tc05_min_tiles chunks, chunk launches from there on."""
    layer = _layer(1, nodes, terms, 32)
    nm, nf, em, ef = _buffers(layer, 64)
    params = torch.zeros([1])
    forward, flows = ({"pcb_lse_contract"} if tiles * -(-k // 128) < 6 else {"pcb_pack_weights", "chunks"}
                      for tiles, k in ((-(-nodes // 128), terms), (-(-terms // 128), nodes)))
    chunk_forms = {"pcb_lse_contract_tc05", "pcb_lse_contract_tc05_ws", "pcb_lse_contract_tc05_accum", "pcb_chunk_combine"}
    monkeypatch.setattr(mod.TUNER, "enabled", False)
    for tmem in (False, None):
        monkeypatch.setattr(SumLayer, "tmem", tmem)
        for run, want in ((lambda: layer(nm, em, params, force_use_bf16=True), forward),
                          (lambda: layer.backward(nf, ef, nm, em, params, None, allow_modify_flows=True,
                                                  _flows_modified=True), flows)):
            calls.clear()
            run()
            got = {"chunks" if c in chunk_forms else c for c in calls}
            if tmem is False:
                short = want is flows and nodes <= 128  # flows of few nodes: short tiles
                assert got == ({"pcb_lse_contract_short"} if short else want)
            else:
                assert "pcb_lse_contract" not in got


@pytest.mark.parametrize("chunks", range(1, 20))
@pytest.mark.parametrize("tiles,rows,B", [(1, 128, 64), (6, 128, 512), (200, 128, 512), (1, 64, 64), (40, 32, 200)])
def test_every_cta_of_a_cluster_has_a_chunk(chunks, tiles, rows, B, monkeypatch):
    monkeypatch.setattr(mod, "_num_sms", lambda: 148)
    ks = mod._tmem_ksplit(tiles, rows, chunks, B)
    assert 1 <= ks <= min(chunks, mod.kTmemCluster)
    # one each as long as a cluster has a CTA per chunk (taller tiles need the shared memory)
    assert rows <= 64 or ks == min(chunks, mod.kTmemCluster)


@pytest.mark.parametrize("ld,taken", [(512, True), (1024, True), (1028, False), (8192, False)])
def test_ratio_workspace_is_no_larger_than_the_flows(ld, taken, calls, monkeypatch):
    """The workspace of log f - log m has the row stride of the caller's buffers, so a batch that is
    a few columns of wide rows goes without it."""
    layer = _layer(8, 128, 128, 32)
    monkeypatch.setattr(SumLayer, "ratio_min_values", 0)
    monkeypatch.setattr(mod.TUNER, "enabled", False)
    buf = torch.empty([layer._layer_nid_range[1], ld])[:, :512]
    made = []
    empty = torch.empty
    monkeypatch.setattr(mod.torch, "empty", lambda shape, **kw: (made.append(shape), empty([1, 1]))[1])
    layer.backward(buf, buf, buf, buf, torch.zeros([1]), None)
    assert ("pcb_flow_ratios" in calls) == taken
    assert [s for s in made if list(s)[-1] == ld] == ([[8 * 128, ld]] if taken else [])


@pytest.mark.parametrize("sub_tiles,B,pays", [(480, 32, False), (800, 24, True), (476, 32, False), (119, 48, False), (240, 48, True),
                                              (96, 48, False), (119, 64, True), (60, 64, False), (60, 200, True), (12, 200, False),
                                              (12, 512, True)])
def test_small_batches_keep_the_other_forms(sub_tiles, B, pays, monkeypatch):
    """Slices of 128 samples are offered where they are filled, or there are many (the measured
    cases beside the rule)."""
    monkeypatch.setattr(mod, "_num_sms", lambda: 148)
    assert mod._tmem_pays(sub_tiles, B) == pays
