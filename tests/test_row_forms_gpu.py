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


def _input_layer(variables, nodes, bs, cats, device):
    with juice.set_block_size(bs):
        leaves = [juice.inputs(v, num_node_blocks=nodes // bs, dist=Categorical(num_cats=cats)) for v in range(variables)]
    return juice.InputLayer(leaves, cum_nodes=bs, pc_num_vars=variables).to(device)


@pytest.mark.parametrize("variables,nodes,bs,cats", [(1, 1, 1, 2), (7, 12, 4, 5), (3, 16, 16, 64), (5, 40, 8, 257),
                                                     (300, 64, 32, 30), (2, 8, 8, 1000)])
@pytest.mark.parametrize("keep_zero", [False, True])
@pytest.mark.parametrize("f64", [False, True])
def test_em_forms(variables, nodes, bs, cats, keep_zero, f64, cuda_device, monkeypatch):
    """One node per warp and several: the same FP64 update, sums in another order."""
    layer = _input_layer(variables, nodes, bs, cats, cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(cats + nodes)
    theta = torch.rand(layer.params.shape, generator=gen, device=cuda_device) + 0.01
    theta[torch.rand(theta.shape, generator=gen, device=cuda_device) < 0.2] = 0.0
    flows = torch.rand([max(layer.num_param_flows, 1)], generator=gen, device=cuda_device)
    got = []
    for many in (False, True):
        monkeypatch.setattr(type(layer), "_em_many", staticmethod(lambda n, k: many))
        with torch.no_grad():
            layer.params.copy_(theta)
        layer.init_param_flows(0.0)
        layer.param_flows.copy_(flows)
        if f64:
            layer.init_param_flows_f64()
            layer.param_flows_f64.copy_(flows.double())
        layer.mini_batch_em(step_size=0.3, pseudocount=0.1, keep_zero_params=keep_zero, use_f64_flows=f64)
        got.append(layer.params.clone())
    assert torch.isfinite(got[0]).all()
    # sums of FP64 differ by a few 2^-53, so the rounded results by at most one unit in the last place
    assert torch.all((got[0] - got[1]).abs() <= 2.0 ** -23 * got[0].abs())


def test_em_rule():
    layer = juice.InputLayer
    assert [layer._em_many(n, k) for n, k in ((16383, 64), (16384, 64), (49151, 256), (49152, 256), (10 ** 6, 257))] == \
        [False, True, False, True, False]


# quads of one variable and not, categories in shared memory and not, ragged batches
@pytest.mark.parametrize("variables,nodes,bs,cats,B", [(1, 1, 1, 2, 1), (5, 6, 2, 17, 33), (3, 16, 16, 256, 130), (4, 20, 4, 257, 515),
                                                       (2, 32, 32, 3000, 64)])
def test_value_forms(variables, nodes, bs, cats, B, cuda_device):
    """Eight nodes per CTA and quads of nodes: the same logarithms, to the bit, with missing values and
    categories that do not exist."""
    nat.device_status()
    layer = _input_layer(variables, nodes, bs, cats, cuda_device)
    d = layer._desc(cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(cats + B)
    with torch.no_grad():
        layer.params.copy_(torch.rand(layer.params.shape, generator=gen, device=cuda_device) + 1e-4)
    data = torch.randint(0, cats, [variables, B], generator=gen, device=cuda_device)
    data[0, 0] = cats
    mask = (torch.rand([B, variables], generator=gen, device=cuda_device) < 0.2).to(torch.uint8)
    got = []
    for name in ("pcb_input_cat_fwd", "pcb_input_cat_fwd_quads"):
        nm = torch.full([bs + variables * nodes, B], 3.0, device=cuda_device)
        nat.call(name, nat.ptr(data), B, nat.ptr(layer.params), nat.ptr(d["vids"]), nat.ptr(d["s_pids"]),
                 nat.ptr(d["ncats"]), variables * nodes, bs, nat.ptr(nm), B, B, nat.ptr(mask), variables, 1, nat.stream())
        got.append(nm)
    assert torch.equal(got[0].nan_to_num(nan=9.0), got[1].nan_to_num(nan=9.0))
    assert torch.all(got[0][:bs] == 3.0)
    assert nat.device_status() == (0 if mask[0, 0] else 4)


@pytest.mark.parametrize("variables,nodes,bs,cats,B", [(1, 1, 1, 2, 1), (5, 6, 2, 17, 33), (3, 32, 16, 256, 130), (4, 33, 1, 300, 515),
                                                       (2, 96, 32, 3000, 1100), (1, 4, 4, 45000, 1024)])
@pytest.mark.parametrize("missing", [False, True])
@pytest.mark.parametrize("log", [False, True])
def test_histogram_forms(variables, nodes, bs, cats, B, missing, log, cuda_device, monkeypatch):
    """One node per warp and one per lane: flows per category against FP64, vocabularies of more than
    40,000 categories at a batch of 1024 on the second (the first refuses them)."""
    layer = _input_layer(variables, nodes, bs, cats, cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(cats + B)
    with torch.no_grad():
        layer.params.copy_(torch.rand(layer.params.shape, generator=gen, device=cuda_device) / cats)
    data = torch.randint(0, cats, [variables, B], generator=gen, device=cuda_device)
    nf = torch.rand([bs + variables * nodes, B], generator=gen, device=cuda_device)
    mask = torch.rand([B, variables], generator=gen, device=cuda_device) < 0.2 if missing else None
    flows = nf.double()[bs:].reshape(variables, nodes, B)
    want = torch.zeros([variables, nodes, cats], dtype=torch.float64, device=cuda_device)
    seen = flows if mask is None else flows * (~mask).T[:, None, :]
    want.scatter_add_(2, data[:, None, :].expand(variables, nodes, B), seen)
    if mask is not None:
        theta = layer.params.double().reshape(variables, nodes, cats)
        want += (flows - seen).sum(dim=2, keepdim=True) * theta
    for tiles in (False, True):
        monkeypatch.setattr(type(layer), "_bwd_tiles", staticmethod(lambda *a: tiles))
        layer.init_param_flows(0.0)
        run = lambda: layer.backward(data, nf.log() if log else nf, nf, missing_mask=mask, logspace_flows=log)
        if cats > 40000 and not tiles:
            with pytest.raises(RuntimeError):
                run()
            continue
        run()
        got = layer.param_flows.double().reshape(want.shape)
        # up to B additions rounded once each, the exponential's and logarithm's 2^-21
        assert torch.all((got - want).abs() <= (B * 2.0 ** -24 + (2.0 ** -20 if log else 0.0)) * want + 1e-12)


def test_histogram_rule():
    tiles = juice.InputLayer._bwd_tiles  # nodes of a variable, categories, variables, batch
    assert [tiles(*a) for a in ((31, 4, 64, 512), (32, 64, 784, 512), (32, 64, 1025, 512), (64, 64, 1025, 512),
                                (64, 600, 784, 256), (64, 600, 784, 257), (64, 2000, 64, 512))] == \
        [False, True, False, True, True, False, True]
