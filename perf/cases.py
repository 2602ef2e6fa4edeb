"""The work this framework does for its users, as measurable cases.

A case is one call pattern of the public entry points -- ``fastgl_b200.trainer.Trainer``, ``fastgl_b200.sampler.
FusedMapSampler`` and the ``fastgl`` operators -- on a seeded R-MAT graph of the sizes that ``bench.py`` and the
tests use.  Six kinds:

* ``train``    a training loop over mini-batches (sampling, aggregation, dense layers, loss, backward, Adam)
* ``blocks``   one mini-batch sampled and mapped hop by hop, as the reference's sampler loop does, and staged into the
               fixed buffers that a captured model reads
* ``window``   a window of mini-batches sampled and mapped in one launch
* ``layer0``   the first layer's neighbour means of a window, straight from the feature table
* ``layer``    one layer through the drop-in operators, forward and backward, block CSR rebuilt from the edge list
* ``ordered``  a layer's backward aggregation with a fixed order of additions (bit-reproducible)

``fanouts`` are written input layer first, as the samplers take them.  ``layer`` and ``ordered`` take blocks of a stated
size with the degrees and the hubs of a sampled one, so that their outputs have a shape that the case fixes.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "fastgl-ae_b200"))

import fastgl  # noqa: E402
from fastgl_b200.graphgen import rmat_graph, synthetic_node_data  # noqa: E402
from fastgl_b200.layers import GAT, GCN, GIN, GraphSAGE  # noqa: E402
from fastgl_b200.sampler import FusedMapSampler  # noqa: E402
from fastgl_b200.trainer import Trainer  # noqa: E402

# R-MAT quadrant probabilities: the skewed graph of the sparse configurations, the flatter one of the dense one
SKEW = {"sparse": (0.57, 0.19, 0.19), "dense": (0.45, 0.22, 0.22)}

PRODUCTS = dict(nodes=2_450_000, degree=50.6, graph="sparse")      # the single-GPU benchmark graph, 124 M edges
SMALL = dict(nodes=100_000, degree=20.0, graph="sparse")           # the CPU-runnable configuration
REDDIT = dict(nodes=233_000, degree=492.0, graph="dense")          # the high-degree configuration, 115 M edges


def listed():
    return [
        # The benchmark's training loop: three-layer GraphSAGE, captured step, windows of 16 mini-batches, products on
        # the tensor cores with error compensation, the loss logged every step.
        dict(name="train sage products", kind="train", model="sage", feat=100, hidden=256, classes=47, fanouts="15,10,5",
             batch=1024, window=16, steps=32, dropout=0.5, matmul="3xtf32", **PRODUCTS),
        # The small configuration, one epoch of ten mini-batches, plain float32 products.
        dict(name="train sage small", kind="train", model="sage", feat=128, hidden=256, classes=10, fanouts="15,10,5",
             batch=1024, window=8, steps=10, dropout=0.5, matmul="fp32", **SMALL),
        # The dense configuration: two-layer GCN on 602-float rows (8-byte aligned only), wide fanouts.
        dict(name="train gcn reddit", kind="train", model="gcn", feat=602, hidden=256, classes=41, fanouts="25,10",
             batch=1024, window=8, steps=8, dropout=0.5, matmul="fp32", **REDDIT),
        # The reference's default run: fanout 5,10,15, 8000 seeds, 64 hidden units; GIN, whose input rows are gathered.
        dict(name="train gin default", kind="train", model="gin", feat=100, hidden=64, classes=47, fanouts="5,10,15",
             batch=8000, window=2, steps=2, dropout=0.5, matmul="fp32", **PRODUCTS),
        # The reference's third model: eight attention heads, coefficients with their gradient.
        dict(name="train gat small", kind="train", model="gat", feat=128, hidden=32, classes=10, fanouts="10,5",
             batch=512, window=4, steps=4, dropout=0.5, matmul="fp32", **SMALL),
        # A handful of seeds through the reference-shaped sampler: what a single query costs.
        dict(name="blocks query", kind="blocks", batch=37, fanouts="15,10,5", replace=False, index="int64", **SMALL),
        # The reference's default mini-batch through the same loop.
        dict(name="blocks default", kind="blocks", batch=8000, fanouts="5,10,15", replace=False, index="int64", **PRODUCTS),
        # A window of eight benchmark mini-batches in one launch.
        dict(name="window products", kind="window", batch=1024, window=8, fanouts="15,10,5", replace=False, index="int64",
             **PRODUCTS),
        # Hubs everywhere, wide fanouts, int32 offsets, picks with replacement (the reference's own mode), short batches.
        dict(name="window reddit", kind="window", batch=1000, window=4, fanouts="25,10", replace=True, index="int32", **REDDIT),
        # 1024-float rows (the wide-feature configuration), one GPU's share of the nodes.
        dict(name="layer0 wide", kind="layer0", nodes=1_000_000, degree=12.0, graph="sparse", feat=1024, batch=1024, window=4,
             fanouts="15,10,5", mode="mean"),
        # One hidden GCN layer of a reference user: degrees, CSR, forward_gcn, backward_gcn on a mid-sized block.
        dict(name="layer gcn", kind="layer", op="gcn", n_dst=1024, n_src=3561, n_edges=3690, fanout=5, dim=64, out=64, heads=1),
        # The reproducible backward of the widest inner layer of the benchmark model.
        dict(name="ordered inner", kind="ordered", n_dst=26_292, n_src=172_681, n_edges=374_231, fanout=15, dim=256, mode="mean",
             self_term=True),
    ]


# ------------------------------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, max_edges=80e6):
    if rng.random() < 0.25:
        nodes, degree, graph = _log_int(rng, 20_000, 233_000), rng.uniform(100.0, 400.0), "dense"
    else:
        nodes, degree, graph = _log_int(rng, 20_000, 2_000_000), math.exp(rng.uniform(math.log(8.0), math.log(60.0))), "sparse"
    return dict(nodes=nodes, degree=round(min(degree, max_edges / nodes), 1), graph=graph)


def _draw_dim(rng, lo, hi):
    """Half of the row widths are whole 16-byte vectors, as most feature tables are; the others are anything."""
    d = _log_int(rng, lo, hi)
    return max(4, d // 4 * 4) if rng.random() < 0.5 else d


def _draw_fanouts(rng, hops, most):
    return ",".join(str(rng.randint(3, most)) for _ in range(hops))


def _draw_block(rng):
    """Sizes of a sampled block: most rows have their full fanout, every second to tenth edge finds a node already seen."""
    fanout, n_dst = rng.randint(3, 15), _log_int(rng, 24, 20_000)
    n_edges = int(n_dst * fanout * rng.uniform(0.5, 1.0))
    return dict(n_dst=n_dst, n_src=n_dst + max(1, int(n_edges * rng.uniform(0.35, 0.9))), n_edges=n_edges, fanout=fanout)


def draw(rng):
    kind = rng.choice(["train", "train", "blocks", "window", "layer0", "layer", "ordered"])
    case = dict(kind=kind)
    if kind == "layer":
        op = rng.choice(["gcn", "gin", "gat"])
        heads = rng.choice([1, 2, 4, 8]) if op == "gat" else 1
        dim = _draw_dim(rng, 16, 602) if heads == 1 else heads * rng.randint(4, 64)
        case.update(op=op, dim=dim, out=_draw_dim(rng, 16, 256), heads=heads, **_draw_block(rng))
        return case
    if kind == "ordered":
        case.update(dim=_draw_dim(rng, 16, 602), mode=rng.choice(["mean", "sum"]), self_term=rng.random() < 0.5, **_draw_block(rng))
        return case
    case.update(_draw_graph(rng))
    batch = _log_int(rng, 24, min(2048, case["nodes"] // 20))
    if kind == "train":
        model = rng.choice(["sage", "sage", "gcn", "gin", "gat"])
        heads = model == "gat"
        hops = 2 if heads else rng.choice([2, 3])
        case.update(model=model, feat=_draw_dim(rng, 32, 256), hidden=_log_int(rng, 8, 32) if heads else _draw_dim(rng, 32, 256),
                    classes=rng.randint(2, 60), fanouts=_draw_fanouts(rng, hops, 12), batch=max(64, batch // 2),
                    window=rng.choice([4, 8]), steps=rng.randint(2, 4) if heads else rng.randint(4, 8), dropout=rng.choice([0.0, 0.5]),
                    matmul=rng.choice(["fp32", "3xtf32"]) if model == "sage" else "fp32")
    elif kind == "blocks":
        case.update(batch=batch, fanouts=_draw_fanouts(rng, rng.choice([1, 2, 3]), 15), replace=rng.random() < 0.3,
                    index=rng.choice(["int32", "int64"]))
    elif kind == "window":
        case.update(batch=batch, window=rng.randint(2, 8), fanouts=_draw_fanouts(rng, rng.choice([2, 3]), 15),
                    replace=rng.random() < 0.3, index=rng.choice(["int32", "int64"]))
    else:
        feat = _draw_dim(rng, 32, 1024)
        case.update(nodes=min(case["nodes"], 1_000_000_000 // feat), feat=feat, batch=min(batch, 1024), window=rng.randint(2, 8),
                    fanouts=_draw_fanouts(rng, 2, 15), mode=rng.choice(["mean", "sum"]))
    return case


# ------------------------------------------------------------------------------------------------------------------
def _fanouts(case):
    return [int(f) for f in case["fanouts"].split(",")]


def _graph(case, seed, dev):
    a, b, c = SKEW[case["graph"]]
    indptr, indices = rmat_graph(case["nodes"], case["degree"], seed=seed, device=dev, a=a, b=b, c=c)
    if case.get("index") == "int32":
        indptr = indptr.to(torch.int32)
    return indptr, indices


def _sampler(case, seed, dev):
    indptr, indices = _graph(case, seed, dev)
    sampler = FusedMapSampler(_fanouts(case), replace=case.get("replace", False), rng_seed=seed)
    sampler.edge_src, sampler.edge_ptr, sampler.nodes_num = indices, indptr, case["nodes"]
    return sampler


def _seed_rows(case, seed, dev, rows):
    """``rows`` mini-batches of distinct seeds, as a shuffled epoch hands them out."""
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed + 17)
    return torch.stack([torch.randperm(case["nodes"], generator=gen, device=dev)[: case["batch"]] for _ in range(rows)]).to(torch.int32)


def _randn(seed, dev, *shape):
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    return torch.randn(shape, generator=gen, device=dev)


class _Training:
    """A trainer as a user's program keeps it; dropping it releases the captured step."""

    def __init__(self, trainer, steps):
        self.trainer, self.steps = trainer, steps

    def __del__(self):
        self.trainer.release_peers()


def _prepare_train(case, seed, dev):
    indptr, indices = _graph(case, seed, dev)
    feat, labels, train = synthetic_node_data(case["nodes"], case["feat"], case["classes"], 0.10, seed=seed, device=dev)
    if train.numel() < case["batch"]:
        train = torch.arange(case["nodes"], dtype=torch.int32, device=dev)
    torch.manual_seed(seed)
    layers = len(_fanouts(case))
    if case["model"] == "sage":
        model = GraphSAGE(case["feat"], case["hidden"], case["classes"], layers, dropout=case["dropout"])
    elif case["model"] == "gat":
        model = GAT(case["feat"], case["hidden"], case["classes"], layers, dropout=case["dropout"], attention_grad=True)
    else:
        model = {"gcn": GCN, "gin": GIN}[case["model"]](case["feat"], case["hidden"], case["classes"], layers, dropout=case["dropout"])
    trainer = Trainer(indptr, indices, feat, labels, train, model.to(dev), _fanouts(case), batch_size=case["batch"],
                      window=case["window"], lr=1e-3, rng_seed=seed, cuda_graph=case["model"] == "sage", matmul=case["matmul"])
    trainer.prime()
    return _Training(trainer, case["steps"])


def _block(case, seed, dev):
    """(row degrees, source ids, destination ids) of a block: rows of 1 .. fanout edges, n_edges in all; every source
    behind the destinations has an edge, the other picks fall on sources of log-normal weight (the degrees that R-MAT
    gives); sources numbered by first occurrence."""
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    n_dst, n_src, n_edges, fanout = case["n_dst"], case["n_src"], case["n_edges"], case["fanout"]
    # n_edges of the n_dst * fanout places: a share of the rows stays below its fanout
    order = torch.argsort(torch.rand(n_dst * fanout, generator=gen, device=dev) *
                          (torch.rand(n_dst, generator=gen, device=dev) + 0.05).repeat_interleave(fanout))
    deg = torch.bincount(order[:n_edges] // fanout, minlength=n_dst)
    weight = torch.exp(2.3 * torch.randn(n_src, generator=gen, device=dev).double())
    below = torch.cumsum(weight, 0)
    new = torch.arange(n_dst, n_src, device=dev)
    drawn = torch.rand(n_edges - new.numel(), generator=gen, device=dev).double() * below[-1]
    src = torch.cat([new, torch.searchsorted(below, drawn).clamp(max=n_src - 1)])
    src = src[torch.randperm(n_edges, generator=gen, device=dev)]
    first = torch.full((n_src,), n_edges, device=dev).scatter_reduce(0, src, torch.arange(n_edges, device=dev), "amin")
    local = torch.arange(n_src, device=dev)
    local[n_dst + torch.argsort(first[n_dst:])] = new
    dst = torch.repeat_interleave(torch.arange(n_dst, device=dev), deg, output_size=n_edges)
    return deg, local[src].to(torch.int32), dst.to(torch.int32)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    kind = case["kind"]
    if kind == "train":
        return _prepare_train(case, seed, dev)
    state = {"case": case}
    if kind == "blocks":
        state["sampler"] = _sampler(case, seed, dev)
        state["seeds"] = _seed_rows(case, seed, dev, 1)[0]
        fanouts = _fanouts(case)
        caps = fastgl.fused_capacity(case["nodes"], case["batch"], fanouts[::-1])
        state["counts"] = torch.zeros(8, dtype=torch.int32, device=dev)
        state["nodes"] = torch.zeros(caps[-1], dtype=torch.int32, device=dev)
        state["blocks"] = [tuple(torch.zeros(n, dtype=torch.int32, device=dev) for n in (cap + 1, cap * f, cap * f))
                           for cap, f in zip(caps[-2::-1], fanouts)]
    elif kind == "window":
        state["sampler"] = _sampler(case, seed, dev)
        state["seeds"] = _seed_rows(case, seed, dev, case["window"])
        counts = [case["batch"]] * case["window"]
        counts[-1] = max(1, case["batch"] * 2 // 3)        # the last mini-batch of an epoch is short
        state["counts"] = torch.tensor(counts, dtype=torch.int32, device=dev)
        # the sampler keeps its result buffers per geometry; what lies behind the counts is zero
        fb = state["sampler"].sample_window(state["seeds"], state["counts"])
        for t in (fb.nodes, *fb.block_indptr, *fb.block_src):
            t.zero_()
    elif kind == "layer0":
        sampler = _sampler(case, seed, dev)
        seeds = _seed_rows(case, seed, dev, case["window"])
        fb = sampler.sample_window(seeds, torch.full((case["window"],), case["batch"], dtype=torch.int32, device=dev))
        fb.counts_host()
        rows = int(1.25 * case["window"] * _expected_blocks(case)[-1][0]) + 8192
        state.update(fb=fb, hop=len(_fanouts(case)) - 1, feat=_randn(seed + 1, dev, case["nodes"], case["feat"]),
                     buf=torch.zeros((rows, 2 * case["feat"]), device=dev))
    elif kind == "layer":
        _, src, dst = _block(case, seed, dev)
        n_src, n_dst = case["n_src"], case["n_dst"]
        state.update(src=src, dst=dst, x=_randn(seed + 1, dev, n_src, case["dim"]))
        if case["op"] == "gat":
            state["weight"] = _randn(seed + 2, dev, src.numel(), case["heads"]).sigmoid()
            state["dy"] = _randn(seed + 3, dev, n_dst, case["dim"])
        else:
            state["weight"] = _randn(seed + 2, dev, case["dim"], case["out"]) / math.sqrt(case["dim"])
            state["dy"] = _randn(seed + 3, dev, n_dst, case["out"])
    else:
        deg, src, _ = _block(case, seed, dev)
        n_src, n_dst = case["n_src"], case["n_dst"]
        indptr = torch.zeros(n_dst + 1, dtype=torch.int32, device=dev)
        indptr[1:] = torch.cumsum(deg, 0)
        state.update(indptr=indptr, src=src, dy=_randn(seed + 1, dev, n_dst, case["dim"]),
                     tb=fastgl.TransposedBlock(n_src, src.numel(), dev), dx=torch.zeros((n_src, case["dim"]), device=dev))
        state["d_self"] = _randn(seed + 2, dev, n_dst, case["dim"]) if case["self_term"] else None
    return state


def run(state):
    if isinstance(state, _Training):
        losses = state.trainer.run_steps(state.steps, read_loss_each_step=True)
        params = list(state.trainer.model.parameters())
        return {"loss": losses, "parameters": [p.detach() for p in params], "gradients": [p.grad for p in params]}
    case = state["case"]
    kind = case["kind"]
    if kind == "blocks":
        # every pass is the mini-batch of the same call counter, so that passes can be compared
        state["sampler"].batch_counter = 0
        input_nodes, _, blocks = state["sampler"].sample_blocks(None, state["seeds"])
        copies = [(state["nodes"], input_nodes)]
        for fixed, b in zip(state["blocks"], blocks):
            copies += zip(fixed, (b.indptr, *b.edges()))
        fastgl.stage_segments(copies[:8], state["counts"], [input_nodes.numel()] + [b.num_edges() for b in blocks])
        if len(copies) > 8:
            fastgl.stage_segments(copies[8:])
        return [state["counts"], state["nodes"], state["blocks"]]
    if kind == "window":
        state["sampler"].batch_counter = 0
        fb = state["sampler"].sample_window(state["seeds"], state["counts"])
        fb.start_readback()
        fb.counts_host()         # the user sizes the next launches from the counts
        return [fb.nodes, fb.counts, *fb.block_indptr, *fb.block_src]
    if kind == "layer0":
        mode = fastgl.AGG_MEAN if case["mode"] == "mean" else fastgl.AGG_SUM
        dim, buf = case["feat"], state["buf"]
        fastgl.aggregate_window(mode, state["fb"], state["hop"], state["feat"], buf[:, dim:], self_out=buf[:, :dim])
        return buf
    if kind == "layer":
        return _run_layer(case, state)
    mode = fastgl.AGG_MEAN if case["mode"] == "mean" else fastgl.AGG_SUM
    tb = fastgl.transpose_block(state["indptr"], state["src"], case["n_dst"], case["n_src"], out=state["tb"])
    return fastgl.aggregate_backward(mode, state["indptr"], state["src"], state["dy"], case["n_src"], d_self=state["d_self"],
                                     out=state["dx"], transposed=tb)


def _run_layer(case, s):
    """What the reference's layers call: block CSR from the edge list, forward operator, backward operator."""
    n_dst, n_src = case["n_dst"], case["n_src"]
    in_degs = fastgl.cal_deg(s["dst"], n_dst)
    edge_ptr = fastgl.exclusive_sum(in_degs)
    fanout = case["fanout"]
    if case["op"] == "gcn":
        dst_degs = in_degs.clamp(min=1)
        src_degs = fastgl.cal_deg(s["src"], n_src).clamp(min=1)
        out = fastgl.forward_gcn(edge_ptr, s["src"], src_degs, dst_degs, s["x"], s["weight"], fanout, n_dst)
        return out + fastgl.backward_gcn(edge_ptr, s["src"], dst_degs, src_degs, s["dy"], s["weight"], s["x"])
    if case["op"] == "gin":
        out = fastgl.forwaed_gin(edge_ptr, s["src"], s["x"], s["weight"], fanout, n_dst)
        return out + fastgl.backward_gin(edge_ptr, s["src"], s["dy"], s["weight"], out[1], n_src)
    out = fastgl.forward_gat(edge_ptr, s["weight"], s["src"], s["x"], fanout, n_dst, case["heads"])
    out = out + fastgl.backward_gat(edge_ptr, s["weight"], s["src"], s["dy"], n_src, case["heads"])
    return out + [fastgl.edge_weight_grad(edge_ptr, s["src"], s["x"], s["dy"], case["heads"])]


# ------------------------------------------------------------------------------------------------------------------
def _expected_blocks(case):
    """Expected (destinations, sources, edges) of every hop of one mini-batch, in sampling order.

    An R-MAT edge puts a node's id together bit by bit, so an id with i ones carries a share p0^(L-i) p1^i of all edge
    endpoints (the ids beyond the last node are folded back; their mass is spread in proportion here): a node's degree
    follows from it, and so does the chance that a pick hits it (the two ends of an edge are nearly independent at
    these quadrant probabilities).  Per hop, every frontier node of degree d gives min(d, fanout) edges, and the nodes
    of each class that are still unseen are thinned out by them."""
    a, b, c = SKEW[case["graph"]]
    n = case["nodes"]
    levels = max(1, math.ceil(math.log2(n)))
    p1 = 1 - a - (b + c) / 2
    p0 = 1 - p1
    size = [0.0] * (levels + 1)                      # nodes by the number of ones in their id
    ones = 0
    for bit in reversed(range(levels + 1)):
        if n >> bit & 1:                             # the ids that agree with n above this bit and have a zero here
            for i in range(bit + 1):
                size[ones + i] += math.comb(bit, i)
            ones += 1
    own = [p0 ** (levels - i) * p1 ** i for i in range(levels + 1)]
    below = sum(s * q for s, q in zip(size, own))
    share = [q / below for q in own]                 # of the endpoints, per node
    degree = [n * case["degree"] * s for s in share]

    def edges_of(mean, fanout):          # E[min(Poisson(mean), fanout)]
        if mean > 8 * fanout:
            return float(fanout)
        p, below, total = math.exp(-mean), 0.0, 0.0
        for k in range(fanout):
            total += k * p
            below += p
            p *= mean / (k + 1)
        return total + fanout * (1.0 - below)

    seen = [case["batch"] * s / n for s in size]
    out = []
    for fanout in reversed(_fanouts(case)):
        edges = sum(u * edges_of(d, fanout) for u, d in zip(seen, degree))
        after = [s - (s - u) * math.exp(-edges * q) for s, u, q in zip(size, seen, share)]
        out.append((sum(seen), sum(after), edges))
        seen = after
    return out


def _sampling_bytes(blocks):
    """Per destination: its id, two offsets and one block offset; per edge: a neighbour id read, a local id written;
    per new node: its id written."""
    return sum(4 * d + 16 * d + 4 * d + 8 * e + 4 * (s - d) for d, s, e in blocks)


def _aggregate_bytes(block, dim, extra_rows=0.0):
    d, s, e = block
    return 4.0 * dim * (s + d + extra_rows) + 4 * e + 4 * d


def work(case):
    """Bytes and operations of one pass: every input read once, every output written once."""
    kind = case["kind"]
    if kind in ("layer", "ordered"):
        blocks = [(case["n_dst"], case["n_src"], case["n_edges"])]
    else:
        blocks = _expected_blocks(case)
    if kind == "blocks":
        # beside the sampling: the destination ids, and the staged copy of everything
        staged = 4 * blocks[-1][1] + sum(4 * d + 8 * e for d, _, e in blocks)
        return {"bytes": _sampling_bytes(blocks) + sum(4 * e for _, _, e in blocks) + 2 * staged, "flops": 0.0}
    if kind == "window":
        return {"bytes": case["window"] * _sampling_bytes(blocks), "flops": 0.0}
    last = blocks[-1]
    if kind == "layer0":
        w = case["window"]
        return {"bytes": w * _aggregate_bytes(last, case["feat"], extra_rows=last[0]), "flops": w * last[2] * case["feat"]}
    if kind == "ordered":
        d, s, e = last
        return {"bytes": _aggregate_bytes(last, case["dim"], extra_rows=d if case["self_term"] else 0), "flops": e * case["dim"]}
    if kind == "layer":
        d, s, e = last
        k, m = case["dim"], case["out"]
        if case["op"] == "gat":
            h = case["heads"]
            return {"bytes": 4.0 * k * (2 * s + 2 * d) + 8 * e + 8 * h * e, "flops": 6.0 * e * k}
        if case["op"] == "gcn":   # x, dx [s, k]; out, dy [d, m]; weight and its gradient
            return {"bytes": 4.0 * (2 * s * k + 2 * d * m + 2 * k * m) + 8 * e, "flops": 6.0 * s * k * m + 4.0 * e * m}
        return {"bytes": 4.0 * (2 * s * k + d * k + 2 * d * m + 2 * k * m) + 8 * e, "flops": 6.0 * d * k * m + 4.0 * e * k}
    # training: sampling, then per layer (input layer first) aggregation and products, forward and backward
    heads = 8 if case["model"] == "gat" else 1
    layers = len(blocks)
    dims = [case["feat"]] + [case["hidden"] * heads] * (layers - 1) + [case["classes"]]
    total, flops = _sampling_bytes(blocks), 0.0
    for i, (d, s, e) in enumerate(reversed(blocks)):
        k, m = dims[i], dims[i + 1]
        kk = 2 * k if case["model"] == "sage" else k
        backward = 0 if i == 0 else 1
        rows = s if case["model"] == "gat" else d
        total += 4.0 * k * s * (1 + backward) + 4.0 * d * m * 2 + 4 * e * (1 + backward)
        flops += 2.0 * rows * kk * m * (2 + backward) + e * k * (1 + backward)
        total += 4.0 * kk * m * 7          # weight, gradient and both moments: read, and written back
    return {"bytes": case["steps"] * total, "flops": case["steps"] * flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("blocks", "window"):
        return "exact"
    if kind == "train":
        # float32 sums in another order move a gradient by 1e-6 of its size; Adam's normalised step turns that into a part
        # of the step size where a gradient is near zero, and the next steps' gradients follow
        return {"rel": 1e-4, "max": 0.1}
    # float32 sums of a few thousand terms at most
    return {"rel": 1e-5, "max": 1e-4}
