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
