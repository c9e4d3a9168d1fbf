"""Row kernels (product layers, Categorical inputs) at the edges of their launch shapes: one
and four rows per thread, rows that take 16-byte accesses and rows that do not, the last
rows of a block, the last samples of a warp."""

import pytest
import torch

import pyjuice_b200 as juice
from pyjuice_b200.nodes.distributions import Categorical

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vectors,nodes,bs,arity,B", [(2, 8, 8, 2, 1), (3, 6, 2, 3, 33), (600, 64, 32, 2, 130),
                                                      (900, 48, 16, 9, 256), (700, 84, 4, 2, 257)])
def test_prod_rows(vectors, nodes, bs, arity, B, cuda_device):
    """Forward values and both backward forms equal the same sums taken in the same order."""
    with juice.set_block_size(bs):
        leaves = [juice.inputs(v, num_node_blocks=nodes // bs, dist=Categorical(num_cats=2)) for v in range(vectors * arity)]
        prods = [juice.multiply(*leaves[r * arity:(r + 1) * arity]) for r in range(vectors)]
    juice.InputLayer(leaves, cum_nodes=bs)
    layer = juice.ProdLayer(prods).to(cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(vectors + B)
    nm = torch.randn([bs + vectors * arity * nodes, B], generator=gen, device=cuda_device)
    em = torch.full([bs + vectors * nodes, B], 7.0, device=cuda_device)
    layer(nm, em)
    rows = nm[bs:].reshape(vectors, arity, nodes, B)
    ref = torch.zeros([vectors, nodes, B], device=cuda_device)
    for j in range(arity):
        ref += rows[:, j]
    assert torch.equal(em[bs:], ref.reshape(-1, B))
    assert torch.all(em[:bs] == 7.0)
    ef = torch.rand([bs + vectors * nodes, B], generator=gen, device=cuda_device)
    spread = ef[bs:].reshape(vectors, 1, nodes, B).expand(vectors, arity, nodes, B).reshape(-1, B)
    for accumulate in (False, True):
        layer.bk_accumulate = accumulate
        nf = torch.ones_like(nm)
        layer.backward(nf, ef)
        assert torch.equal(nf[bs:], spread + (1.0 if accumulate else 0.0))
        assert torch.all(nf[:bs] == 1.0)


@pytest.mark.parametrize("bs,blocks,cats,B", [(1, 1, 2, 1), (2, 3, 5, 37), (4, 3, 256, 130), (8, 4, 257, 64), (16, 2, 64, 1023)])
def test_input_values(bs, blocks, cats, B, cuda_device):
    """Values, summed-out samples and the NaN of an impossible category, for variables whose
    nodes straddle the kernel's groups of nodes."""
    with juice.set_block_size(bs):
        leaves = [juice.inputs(v, num_node_blocks=blocks, dist=Categorical(num_cats=cats)) for v in range(5)]
    layer = juice.InputLayer(leaves, cum_nodes=bs, pc_num_vars=5).to(cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(B)
    n = bs * blocks
    theta = torch.rand([5, n, cats], generator=gen, device=cuda_device) + 0.01
    with torch.no_grad():
        layer.params.copy_(theta.reshape(-1))
    data = torch.randint(0, cats, [5, B], generator=gen, device=cuda_device)
    mask = torch.rand([B, 5], generator=gen, device=cuda_device) < 0.3
    ref = theta.double().log().gather(2, data[:, None, :].expand(5, n, B))
    nm = torch.full([bs + 5 * n, B], 3.0, device=cuda_device)
    layer(data, nm)
    # __logf: absolute error 2^-21.4 in [0.5, 2], 3 ulp of the result outside
    assert torch.all((nm[bs:].double() - ref.reshape(-1, B)).abs() <= 4e-7 + 4e-7 * ref.reshape(-1, B).abs())
    assert torch.all(nm[:bs] == 3.0)
    full = nm.clone()
    layer(data, nm, missing_mask=mask)
    gone = mask.T[:, None, :].expand(5, n, B).reshape(-1, B)
    assert torch.equal(nm[bs:], torch.where(gone, torch.zeros_like(full[bs:]), full[bs:]))
    data[2, B // 2] = cats
    layer(data, nm)
    bad = torch.zeros([5, n, B], dtype=torch.bool, device=cuda_device)
    bad[2, :, B // 2] = True
    assert torch.equal(torch.isnan(nm[bs:]), bad.reshape(-1, B))
    from pyjuice_b200 import _native as nat
    assert nat.device_status(clear=True) == 4


@pytest.mark.parametrize("nodes,cats,B,missing", [(1, 2, 1, False), (16, 3, 513, True), (32, 64, 512, False),
                                                  (48, 300, 1030, True), (96, 7000, 700, False)])
def test_input_flows_and_em(nodes, cats, B, missing, cuda_device):
    """Flow histogram (added to what the slots hold) and EM against FP64: one sample, more
    samples than one chunk, fewer nodes than a tile, every node in one category, vocabularies
    beyond a batch."""
    with juice.set_block_size(1):
        leaves = [juice.inputs(v, num_node_blocks=nodes, dist=Categorical(num_cats=cats)) for v in range(3)]
    layer = juice.InputLayer(leaves, cum_nodes=1, pc_num_vars=3).to(cuda_device)
    gen = torch.Generator(device=cuda_device).manual_seed(cats)
    theta = torch.rand([3, nodes, cats], generator=gen, device=cuda_device) + 0.01
    theta = theta / theta.sum(dim=2, keepdim=True)
    data = torch.randint(0, cats, [3, B], generator=gen, device=cuda_device)
    data[0] = cats - 1
    mask = torch.rand([B, 3], generator=gen, device=cuda_device) < 0.4 if missing else None
    nf = torch.rand([1 + 3 * nodes, B], generator=gen, device=cuda_device)
    old = torch.rand([3, nodes, cats], generator=gen, device=cuda_device)
    with torch.no_grad():
        layer.params.copy_(theta.reshape(-1))
    layer.init_param_flows(flows_memory=0.0)
    layer.param_flows.copy_(old.reshape(-1))
    layer.backward(data, nf, torch.zeros_like(nf), missing_mask=mask)
    f = nf[1:].reshape(3, nodes, B).double()
    gone = torch.zeros([3, nodes, B], dtype=torch.bool, device=cuda_device)
    if missing:
        gone = mask.T[:, None, :].expand(3, nodes, B)
    ref = old.double().scatter_add(2, data[:, None, :].expand(3, nodes, B), torch.where(gone, 0.0, f))
    ref += torch.where(gone, f, 0.0).sum(dim=2, keepdim=True) * theta.double()
    got = layer.param_flows.reshape(3, nodes, cats).double()
    # sums of at most B + 2 positive terms in FP32: relative error (B + 2) 2^-24
    assert torch.all((got - ref).abs() <= (B + 2) * 2.0 ** -24 * ref)
    layer.mini_batch_em(step_size=0.3, pseudocount=0.1)
    new = 0.7 * theta.double() + 0.3 * (got + 0.1 / cats) / (got.sum(dim=2, keepdim=True) + 0.1)
    # FP64 arithmetic rounded once to FP32
    assert torch.all((layer.params.reshape(3, nodes, cats).double() - new).abs() <= 2.0 ** -23 * new)
