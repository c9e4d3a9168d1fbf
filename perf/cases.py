"""The work that programs built on this framework have it do, as measurable cases.

Five kinds, each through a public entry point:

* ``step``: one mini-batch EM step of a compiled HCLT (forward, ``lls.mean().backward()``,
  ``mini_batch_em``), the inner loop of training; returns the log-likelihoods and the
  updated parameters.
* ``likelihood``: log-likelihoods of token sequences under a compiled HMM, the inner loop of
  evaluation.
* ``sum``: one sum layer alone, forward (node values) or backward (element flows and
  parameter flows). Dense regions are what HCLT and PD levels and HMM transitions are made
  of; ``density`` below 1 keeps a random part of the blocks.
* ``prod``: one product layer alone, forward or backward.
* ``input``: one Categorical input layer alone: its forward, or its flows and EM update.

A case names sizes only. Whatever has to be the same for every seed (the tree of an HCLT,
the kept blocks of a sparse layer) is drawn from the sizes; parameters, values, flows and
data are drawn from the seed. ``fp32`` asks for the plain FP32 form, otherwise the default
rule picks the tensor-core form where it applies.
"""

from __future__ import annotations

import copy
import functools
import random

import torch

import pyjuice_b200 as juice
from pyjuice_b200.nodes.distributions import Categorical
from pyjuice_b200.structures import HMM, hclt_from_tree

DEVICE = "cuda:0"
STEP_SIZE = 0.1
PSEUDOCOUNT = 0.1


def listed():
    return [
        # A training step of a small model at a small batch: every launch is tiny, so what
        # counts is how many there are and what the host does between them.
        _step("step_hclt64", 64, 4, 16, 16, 64, False),
        # The training step of the headline benchmark: 28 x 28 pixels, 256 grey levels.
        _step("step_hclt784", 784, 256, 128, 32, 512, False),
        # Perplexity of a language-model-sized vocabulary under a 512-state HMM.
        _likelihood("likelihood_hmm512", 32, 512, 33279, 512, False),
        # A level of 200 dense 256 x 256 regions, forward and backward.
        _sum("sum_fwd_200x256", 200, 256, 256, 32, 512, False, "fwd", 1.0),
        _sum("sum_bwd_200x256", 200, 256, 256, 32, 512, False, "bwd", 1.0),
        # The largest level of the 128-latent HCLT in plain FP32, and a mid-sized one at an
        # odd batch (the last batch of an epoch).
        _sum("sum_fwd_fp32_119x128", 119, 128, 128, 32, 512, True, "fwd", 1.0),
        _sum("sum_bwd_fp32_25x96", 25, 96, 96, 32, 237, True, "bwd", 1.0),
        # Block-sparse sums: 1024 nodes over 1024 children, a fifth of the 32 x 32 blocks.
        _sum("sum_fwd_sparse_16x1024", 16, 1024, 1024, 32, 512, False, "fwd", 0.2),
        # One HMM transition of 2048 states for a batch of 64 sequences, flows included.
        _sum("sum_bwd_hmm2048", 1, 2048, 2048, 32, 64, False, "bwd", 1.0),
        # The product level below 200 regions of 256 nodes.
        _prod("prod_fwd_200x256", 200, 256, 2, 16, 512, "fwd"),
        # Inputs: 784 variables x 256 nodes, 64 categories; values, then flows and EM.
        _input("input_fwd_784x256", 784, 256, 64, 512, "fwd"),
        _input("input_em_784x256", 784, 256, 64, 512, "em"),
    ]


def _step(name, num_vars, cats, latents, block, batch, fp32):
    return dict(name=name, kind="step", num_vars=num_vars, cats=cats, latents=latents, block=block, batch=batch,
                fp32=fp32)


def _likelihood(name, length, latents, vocab, batch, fp32):
    return dict(name=name, kind="likelihood", length=length, latents=latents, vocab=vocab, batch=batch, fp32=fp32)


def _sum(name, regions, latents, terms, block, batch, fp32, direction, density):
    return dict(name=name, kind="sum", regions=regions, latents=latents, terms=terms, block=block, batch=batch,
                fp32=fp32, direction=direction, density=density)


def _prod(name, vectors, nodes, arity, block, batch, direction):
    return dict(name=name, kind="prod", vectors=vectors, nodes=nodes, arity=arity, block=block, batch=batch,
                direction=direction)


def _input(name, num_vars, nodes, cats, batch, direction):
    return dict(name=name, kind="input", num_vars=num_vars, nodes=nodes, cats=cats, batch=batch, direction=direction)


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))

    kind = rng.choice(("sum", "sum", "sum", "sum", "prod", "input", "step", "likelihood"))
    batch = log_int(16, 512)
    fp32 = rng.random() < 0.35
    if kind == "sum":
        block = rng.choice((16, 32, 64))
        latents = block * log_int(1, 1024 // block)
        terms = block * log_int(1, 1024 // block)
        regions = log_int(1, max(1, min(200, 13_000_000 // (latents * terms))))
        density = 0.2 if latents >= 8 * block and terms >= 8 * block and rng.random() < 0.4 else 1.0
        case = _sum("", regions, latents, terms, block, batch, fp32, rng.choice(("fwd", "bwd")), density)
    elif kind == "prod":
        block = rng.choice((16, 32))
        case = _prod("", log_int(4, 200), block * log_int(1, 256 // block), rng.randint(2, 4), block, batch,
                     rng.choice(("fwd", "bwd")))
    elif kind == "input":
        case = _input("", log_int(16, 784), 16 * log_int(1, 16), log_int(2, 256), batch, rng.choice(("fwd", "em")))
    elif kind == "step":
        latents = 16 * log_int(1, 8)
        case = _step("", log_int(4, 14) ** 2, log_int(2, 256), latents, 16 if latents % 32 else 32, batch, fp32)
    else:
        case = _likelihood("", rng.randint(8, 32), 32 * log_int(1, 16), log_int(64, 33279), batch, fp32)
    del case["name"]
    return case


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, _generator(case, seed))


def run(state):
    return state["run"]()


def work(case):
    return _KINDS[case["kind"]][1](case)


def exact(case, seed):
    return _KINDS[case["kind"]][2](case, _generator(case, seed))


def _generator(case, seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _rand(gen, *shape):
    return torch.rand(shape, generator=gen, device=DEVICE)


def _randn(gen, *shape):
    return torch.randn(shape, generator=gen, device=DEVICE)


def _simplex(gen, *shape, dim):
    """Random weights that sum to one over ``dim`` (the library's own initial spread)."""
    w = torch.exp(-4.0 * _rand(gen, *shape))
    return w / w.sum(dim=dim, keepdim=True)


# ---------------------------------------------------------------- step: EM of an HCLT

@functools.lru_cache(maxsize=None)
def _grid_tree(num_vars):
    """Children, post-order and root of a random spanning tree of a pixel grid (what a Chow-Liu
    tree of images looks like), rooted at the middle of its longest path as HCLT does."""
    rng = random.Random(num_vars)
    side = int(round(num_vars ** 0.5))
    edges = []
    for v in range(num_vars):
        if v % side + 1 < side and v + 1 < num_vars:
            edges.append((rng.random(), v, v + 1))
        if v + side < num_vars:
            edges.append((rng.random(), v, v + side))
    parent = list(range(num_vars))

    def find(a):
        while parent[a] != a:
            parent[a] = parent[parent[a]]
            a = parent[a]
        return a

    adjacent = {v: [] for v in range(num_vars)}
    for _, u, v in sorted(edges):
        if find(u) != find(v):
            parent[find(u)] = find(v)
            adjacent[u].append(v)
            adjacent[v].append(u)

    def path_to_farthest(v):
        paths, queue = {v: [v]}, [v]
        for a in queue:
            for b in adjacent[a]:
                if b not in paths:
                    paths[b] = paths[a] + [b]
                    queue.append(b)
        return paths[queue[-1]]

    longest = path_to_farthest(path_to_farthest(0)[-1])
    root = longest[len(longest) // 2]
    children, order, stack = {}, [], [(root, -1)]
    while stack:
        v, p = stack.pop()
        children[v] = [c for c in adjacent[v] if c != p]
        order.append(v)
        stack += [(c, v) for c in children[v]]
    return children, order[::-1], root


@functools.lru_cache(maxsize=1)
def _hclt(num_vars, cats, latents, block):
    """The compiled circuit of an HCLT on the host (each state takes a copy), and per variable
    the sum vector of its region (None for a leaf)."""
    children, order, root = _grid_tree(num_vars)
    ns = hclt_from_tree(order, children, root, latents, input_dist=Categorical(num_cats=cats), block_size=block)
    return juice.compile(ns)


def _step_inputs(case, gen):
    """Parameters as the compiled layout holds them (a sum vector's: per node block, children
    x block), and smooth random images."""
    n, cats, L, bs, B = case["num_vars"], case["cats"], case["latents"], case["block"], case["batch"]
    theta = _simplex(gen, n * L, cats, dim=1)
    weights = _simplex(gen, n, L // bs, L, bs, dim=2)
    top = _simplex(gen, L, dim=0)
    side = int(round(n ** 0.5))
    z = torch.nn.functional.avg_pool2d(_randn(gen, B, 1, side + 4, side + 4), 5, 1).reshape(B, n) * 5.0
    x = (torch.special.ndtr(z) * cats).long().clamp_(0, cats - 1)
    return theta, weights, top, x


def _prepare_step(case, gen):
    theta, weights, top, x = _step_inputs(case, gen)
    n, L = case["num_vars"], case["latents"]
    pc = copy.deepcopy(_hclt(n, case["cats"], L, case["block"])).to(DEVICE)
    layer = pc.input_layer_group[0]
    with torch.no_grad():
        for ns in layer.nodes:
            v = next(iter(ns.scope))
            lo, hi = ns._param_range
            layer.params[lo:hi] = theta[v * L:(v + 1) * L].reshape(-1)
        i = 0
        for ns in pc.root_ns:
            if ns.is_sum():
                lo, hi = ns._param_range
                pc.params[lo:hi] = top if ns is pc.root_ns else weights[i].reshape(-1)
                i += 1
    kw = dict(force_use_fp32=True) if case["fp32"] else {}

    def step():
        pc.init_param_flows(flows_memory=0.0)
        lls = pc(x, record_cudagraph=True, **kw)
        lls.mean().backward()
        pc.mini_batch_em(step_size=STEP_SIZE, pseudocount=PSEUDOCOUNT)
        return dict(lls=lls.detach(), params=pc.params, input_params=layer.params)

    return dict(run=step)


def _step_sizes(case):
    children, _, root = _grid_tree(case["num_vars"])
    inner = sum(1 for v, c in children.items() if c and v != root)
    return inner, inner * case["latents"] ** 2 + case["latents"], case["num_vars"] * case["latents"] * case["cats"]


def _work_step(case):
    _, edges, theta = _step_sizes(case)
    return dict(bytes=8 * case["num_vars"] * case["batch"] + 8 * (edges + theta) + 4 * case["batch"],
                flops=6 * edges * case["batch"])


def _exact_step(case, gen):
    """The log-likelihoods, by one upward pass over the tree. The updated parameters have no
    value here: they are a training step's state, laid out by the compiler."""
    theta, weights, top, x = _step_inputs(case, gen)
    n, L, bs, B = case["num_vars"], case["latents"], case["block"], case["batch"]
    children, order, root = _grid_tree(n)
    logt = theta.double().log().reshape(n, L, case["cats"])
    value, i = {}, 0
    for v in order:
        value[v] = logt[v][:, x[:, v]]
        if children[v]:
            for c in children[v]:
                value[v] = value[v] + value.pop(c)
            m = value[v].amax(dim=0)
            e = torch.exp(value[v] - m)
            if v == root:
                w = top.double()[None, :]
            else:
                w = weights[_sum_index(n)[v]].double().permute(0, 2, 1).reshape(L, L)
            value[v] = torch.log(w @ e) + m
    return dict(lls=value[root].T.contiguous(), params=None, input_params=None)


@functools.lru_cache(maxsize=None)
def _sum_index(num_vars):
    """Position of each region's sum vector among the circuit's sum vectors: children first, in
    the order in which the tree lists them, a node after all of its children."""
    children, _, root = _grid_tree(num_vars)
    index, stack = {}, [(root, False)]
    while stack:
        v, done = stack.pop()
        if done:
            index[v] = len(index)
        elif children[v]:
            stack.append((v, True))
            stack += [(c, False) for c in reversed(children[v])]
    return index


# ---------------------------------------------------------------- likelihood: an HMM

def _likelihood_inputs(case, gen):
    H, V, T, B = case["latents"], case["vocab"], case["length"], case["batch"]
    alpha, gamma = _simplex(gen, H, H, dim=1), _simplex(gen, H, dim=0)
    beta = _simplex(gen, H, V, dim=1)
    # words by rank: frequent ones often, as in text
    x = (V ** _rand(gen, B, T)).long().sub_(1).clamp_(0, V - 1)
    return alpha, beta, gamma, x


def _prepare_likelihood(case, gen):
    alpha, beta, gamma, x = _likelihood_inputs(case, gen)
    ns = HMM(case["length"], case["latents"], case["vocab"], block_size=32, alpha=alpha.cpu(), beta=beta.cpu(),
             gamma=gamma.cpu())
    pc = juice.compile(ns).to(DEVICE)
    kw = dict(force_use_fp32=True) if case["fp32"] else {}

    def evaluate():
        with torch.no_grad():
            return pc(x, record_cudagraph=True, **kw)

    return dict(run=evaluate)


def _work_likelihood(case):
    H, T, B = case["latents"], case["length"], case["batch"]
    used = min(case["vocab"], T * B)
    return dict(bytes=4 * H * H + 4 * H * used + 8 * T * B + 4 * B, flops=2 * H * H * (T - 1) * B)


def _exact_likelihood(case, gen):
    alpha, beta, gamma, x = _likelihood_inputs(case, gen)
    a, g = alpha.double(), gamma.double()
    ll = torch.zeros([case["batch"]], dtype=torch.float64, device=DEVICE)
    state = beta[:, x[:, -1]].double()
    for t in range(case["length"] - 2, -1, -1):
        m = state.amax(dim=0)
        ll += m.log()
        state = (a @ (state / m)) * beta[:, x[:, t]].double()
    return (torch.log(g @ state) + ll)[:, None]


# ---------------------------------------------------------------- sum: one sum layer

@functools.lru_cache(maxsize=1)
def _sum_blocks(latents, terms, block, density):
    """[node blocks, child blocks] of kept blocks, the same in every region; no empty row or column."""
    nb, cb = latents // block, terms // block
    if density >= 1.0:
        return torch.ones([nb, cb], dtype=torch.bool)
    rng = random.Random(latents * 10007 + terms)
    keep = torch.tensor([[rng.random() < density for _ in range(cb)] for _ in range(nb)])
    for i in range(max(nb, cb)):
        keep[i % nb, i % cb] = True
    return keep


def _sum_layer(case):
    R, bs = case["regions"], case["block"]
    nb, cb = case["latents"] // bs, case["terms"] // bs
    edges = _sum_blocks(case["latents"], case["terms"], bs, case["density"]).nonzero().T.contiguous()
    with juice.set_block_size(bs):
        leaves = [juice.inputs(v, num_node_blocks=cb, dist=Categorical(num_cats=2)) for v in range(2 * R)]
        prods = [juice.multiply(leaves[2 * r], leaves[2 * r + 1]) for r in range(R)]
        sums = [juice.summate(p, num_node_blocks=nb, edge_ids=edges) for p in prods]
    juice.InputLayer(leaves, cum_nodes=bs)
    juice.ProdLayer(prods)
    return juice.SumLayer(sums, global_nid_start=bs, global_pid_start=bs ** 2, global_pfid_start=0,
                          node2tiednodes=dict()).to(DEVICE)


def _sum_inputs(case, gen):
    """Weights [R, L, K] (zero where no edge is), element values [R, K, B] (log-probabilities
    of scopes of 1 to about 20 variables), the node values that follow from them, and node
    flows [R, L, B] (each region's flows sum to one in every sample)."""
    R, L, K, bs, B = case["regions"], case["latents"], case["terms"], case["block"], case["batch"]
    keep = _sum_blocks(L, K, bs, case["density"]).to(DEVICE).repeat_interleave(bs, 0).repeat_interleave(bs, 1)
    w = torch.exp(-4.0 * _rand(gen, R, L, K)) * keep
    w = w / w.sum(dim=2, keepdim=True)
    em = 2.0 * _randn(gen, R, K, B) - 3.0 * torch.exp(3.0 * _rand(gen, R, 1, 1)) - 2.0 * _rand(gen, R, 1, B)
    nf = torch.softmax(2.0 * _randn(gen, R, L, B), dim=1)
    return w, em, nf


def _sum_values(w, em):
    """Node values [R, L, B] in 64 bits."""
    out = torch.empty([w.size(0), w.size(1), em.size(2)], dtype=torch.float64, device=DEVICE)
    for r in range(w.size(0)):
        e = em[r].double()
        m = e.amax(dim=0)
        out[r] = torch.log(w[r].double() @ torch.exp(e - m)) + m
    return out


def _sum_pack(case, x):
    """[R, L, K] per edge -> the compiled order: per region and node block its kept child nodes,
    each with its block of nodes."""
    R, L, K, bs = case["regions"], case["latents"], case["terms"], case["block"]
    keep = _sum_blocks(L, K, bs, case["density"]).to(x.device)
    y = x.reshape(R, L // bs, bs, K // bs, bs).permute(0, 1, 3, 4, 2)
    return y[:, keep].reshape(-1)


def _prepare_sum(case, gen):
    w, em, nf = _sum_inputs(case, gen)
    bs, B = case["block"], case["batch"]
    layer = _sum_layer(case)
    params = torch.cat([torch.zeros([bs ** 2], device=DEVICE), _sum_pack(case, w)])
    ems = torch.cat([torch.full([bs, B], -float("inf"), device=DEVICE), em.reshape(-1, B)])
    form = dict(force_use_fp32=True) if case["fp32"] else {}
    rows = bs + case["regions"] * case["latents"]
    if case["direction"] == "fwd":
        nm = torch.zeros([rows, B], device=DEVICE)

        def forward():
            layer(nm, ems, params, **form)
            return nm

        return dict(run=forward)
    nms = torch.zeros([rows, B], device=DEVICE)
    nms[bs:] = _sum_values(w, em).float().reshape(-1, B)
    nfs = torch.zeros([rows, B], device=DEVICE)
    nfs[bs:] = nf.reshape(-1, B)
    ef = torch.zeros_like(ems)
    pf = torch.zeros([params.numel() - bs ** 2], device=DEVICE)

    def backward():
        pf.zero_()
        layer.backward(nfs, ef, nms, ems, params, pf, **form)
        return dict(element_flows=ef, param_flows=pf)

    return dict(run=backward)


def _sum_edges(case):
    keep = _sum_blocks(case["latents"], case["terms"], case["block"], case["density"])
    return case["regions"] * int(keep.sum()) * case["block"] ** 2


def _work_sum(case):
    edges, R, B = _sum_edges(case), case["regions"], case["batch"]
    if case["direction"] == "fwd":
        return dict(bytes=4 * R * (case["latents"] + case["terms"]) * B + 4 * edges, flops=2 * edges * B)
    return dict(bytes=4 * R * 2 * (case["latents"] + case["terms"]) * B + 8 * edges, flops=4 * edges * B)


def _exact_sum(case, gen):
    w, em, nf = _sum_inputs(case, gen)
    R, L, K, bs, B = case["regions"], case["latents"], case["terms"], case["block"], case["batch"]
    nm = _sum_values(w, em)
    if case["direction"] == "fwd":
        out = torch.zeros([bs + R * L, B], dtype=torch.float64, device=DEVICE)
        out[bs:] = nm.reshape(-1, B)
        return out
    nm = nm.float().double()  # the values that the layer is given
    ef = torch.zeros([bs + R * K, B], dtype=torch.float64, device=DEVICE)
    pf = torch.empty([R, L, K], dtype=torch.float64, device=DEVICE)
    for r in range(R):
        e = em[r].double()
        m = e.amax(dim=0)
        ratio = nf[r].double() * torch.exp(m - nm[r])
        e = torch.exp(e - m)
        ef[bs + r * K:bs + (r + 1) * K] = (w[r].double().T @ ratio) * e
        pf[r] = w[r].double() * (ratio @ e.T)
    return dict(element_flows=ef, param_flows=_sum_pack(case, pf))


# ---------------------------------------------------------------- prod: one product layer

def _prod_layer(case):
    bs = case["block"]
    nb = case["nodes"] // bs
    with juice.set_block_size(bs):
        leaves = [juice.inputs(v, num_node_blocks=nb, dist=Categorical(num_cats=2))
                  for v in range(case["vectors"] * case["arity"])]
        prods = [juice.multiply(*leaves[r * case["arity"]:(r + 1) * case["arity"]]) for r in range(case["vectors"])]
    juice.InputLayer(leaves, cum_nodes=bs)
    return juice.ProdLayer(prods).to(DEVICE)


def _prod_inputs(case, gen):
    V, A, N, B = case["vectors"], case["arity"], case["nodes"], case["batch"]
    if case["direction"] == "fwd":
        return -20.0 * _rand(gen, V, A, N, B)
    return torch.softmax(2.0 * _randn(gen, V, N, B), dim=1)


def _prepare_prod(case, gen):
    layer = _prod_layer(case)
    x = _prod_inputs(case, gen)
    V, A, N, B, bs = case["vectors"], case["arity"], case["nodes"], case["batch"], case["block"]
    nodes = torch.zeros([bs + V * A * N, B], device=DEVICE)
    elements = torch.zeros([bs + V * N, B], device=DEVICE)
    if case["direction"] == "fwd":
        nodes[bs:] = x.reshape(-1, B)

        def forward():
            layer(nodes, elements)
            return elements

        return dict(run=forward)
    elements[bs:] = x.reshape(-1, B)

    def backward():
        nodes.zero_()
        layer.backward(nodes, elements)
        return nodes

    return dict(run=backward)


def _work_prod(case):
    rows = case["vectors"] * case["nodes"] * (case["arity"] + 1)
    return dict(bytes=4 * rows * case["batch"], flops=case["vectors"] * case["nodes"] * case["arity"] * case["batch"])


def _exact_prod(case, gen):
    x = _prod_inputs(case, gen).double()
    V, A, N, B, bs = case["vectors"], case["arity"], case["nodes"], case["batch"], case["block"]
    if case["direction"] == "fwd":
        out = torch.zeros([bs + V * N, B], dtype=torch.float64, device=DEVICE)
        out[bs:] = x.sum(dim=1).reshape(-1, B)
    else:
        out = torch.zeros([bs + V * A * N, B], dtype=torch.float64, device=DEVICE)
        out[bs:] = x[:, None].expand(V, A, N, B).reshape(-1, B)
    return out


# ---------------------------------------------------------------- input: one Categorical layer

def _input_layer(case):
    with juice.set_block_size(16):
        leaves = [juice.inputs(v, num_node_blocks=case["nodes"] // 16, dist=Categorical(num_cats=case["cats"]))
                  for v in range(case["num_vars"])]
    return juice.InputLayer(leaves, cum_nodes=16, pc_num_vars=case["num_vars"]).to(DEVICE)


def _input_inputs(case, gen):
    V, N, K, B = case["num_vars"], case["nodes"], case["cats"], case["batch"]
    theta = _simplex(gen, V, N, K, dim=2)
    data = torch.special.ndtr(_randn(gen, V, B) + 0.5 * _randn(gen, V, 1)).mul_(K).long().clamp_(0, K - 1)
    flows = torch.softmax(2.0 * _randn(gen, V, N, B), dim=1)
    return theta, data, flows


def _prepare_input(case, gen):
    layer = _input_layer(case)
    theta, data, flows = _input_inputs(case, gen)
    B = case["batch"]
    with torch.no_grad():
        layer.params.copy_(theta.reshape(-1))
    nm = torch.zeros([16 + case["num_vars"] * case["nodes"], B], device=DEVICE)
    if case["direction"] == "fwd":

        def forward():
            layer(data, nm)
            return nm

        return dict(run=forward)
    nf = torch.zeros_like(nm)
    nf[16:] = flows.reshape(-1, B)

    def update():
        layer.init_param_flows(flows_memory=0.0)
        layer.backward(data, nf, nm)
        layer.mini_batch_em(step_size=STEP_SIZE, pseudocount=PSEUDOCOUNT)
        return dict(param_flows=layer.param_flows, params=layer.params)

    return dict(run=update)


def _work_input(case):
    V, N, K, B = case["num_vars"], case["nodes"], case["cats"], case["batch"]
    if case["direction"] == "fwd":
        return dict(bytes=4 * V * N * (min(K, B) + B) + 8 * V * B, flops=V * N * B)
    return dict(bytes=4 * V * N * (3 * K + B) + 8 * V * B, flops=V * N * (B + 4 * K))


def _exact_input(case, gen):
    theta, data, flows = _input_inputs(case, gen)
    V, N, K, B = case["num_vars"], case["nodes"], case["cats"], case["batch"]
    index = data[:, None, :].expand(V, N, B)
    theta = theta.double()
    if case["direction"] == "fwd":
        out = torch.zeros([16 + V * N, B], dtype=torch.float64, device=DEVICE)
        out[16:] = theta.gather(2, index).log_().reshape(-1, B)
        return out
    pf = torch.zeros([V, N, K], dtype=torch.float64, device=DEVICE).scatter_add_(2, index, flows.double())
    new = (pf + PSEUDOCOUNT / K) / (pf.sum(dim=2, keepdim=True) + PSEUDOCOUNT)
    return dict(param_flows=pf.reshape(-1), params=((1.0 - STEP_SIZE) * theta + STEP_SIZE * new).reshape(-1))


_KINDS = {
    "step": (_prepare_step, _work_step, _exact_step),
    "likelihood": (_prepare_likelihood, _work_likelihood, _exact_likelihood),
    "sum": (_prepare_sum, _work_sum, _exact_sum),
    "prod": (_prepare_prod, _work_prod, _exact_prod),
    "input": (_prepare_input, _work_input, _exact_input),
}
