"""The work this framework is used for, as cases that can be timed: whole mini-batches of every sampling strategy that
one GPU runs, the feature gather by itself, and the sparse layers (forward and backward) over sampled blocks.

A case names its kind:

  batch   one mini-batch: sampler.sample() of one strategy, ops.load_subtensor of its input nodes and the neighbour sums
          (or attention) of every layer, down to one row per seed; a model's own weights are left out
  epoch   several such mini-batches through sampler.sample_iter(), from seeds in page-locked host memory, as a training
          loop takes them
  gather  ops.load_subtensor of distinct ids against a device cache (and, for a share of them, host memory)
  sage    ops.spmm_copy_u_sum over a block and, for the gradient, over the same block with its two sides swapped
  gat     the fused attention layer through autograd: forward, then the gradients of ft, el and er
  edges   the separate edge operators: sddmm_u_add_v, spmm_u_mul_e_sum and sddmm_u_mul_v

The graph and the feature tables of a batch, epoch or gather case are the data set of a training run: they follow from
the case's sizes, are installed once and stay (operators and samplers keep them in the process-wide state); the seed
picks the nodes a mini-batch starts from, the ids of a gather, and all tensors of a layer.
"""
import math

import torch

from apt_b200 import ops, sampler, synthetic

_TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
_BYTES = {"f32": 4, "bf16": 2, "f16": 2}
_SAMPLE_KEY = 2025
# device memory of a cached feature table, and page-locked host memory of a table whose rows then repeat
_CACHE_BYTES = 15 * 10 ** 9
_HOST_BYTES = 1 << 30


def listed():
    small = dict(nodes=1 << 20, edges=16_000_000, undirected=False, dim=128, dtype="f32", cached=0.25)
    return [
        # the smallest mini-batch in use (a small graph, 256 seeds): launches and host work count
        dict(name="np_batch_tiny", kind="batch", strategy="np", nodes=1 << 16, edges=1 << 20, undirected=False, dim=128,
             dtype="f32", cached=0.25, batch=256, fanouts="15,10,5"),
        # the headline configuration: papers-shaped graph, 1024 seeds, three hops, a quarter of the rows cached
        dict(name="np_batch_papers", kind="batch", strategy="np", nodes=111_059_956, edges=1_600_000_000,
             undirected=False, dim=128, dtype="f32", cached=0.25, batch=1024, fanouts="15,10,5"),
        # a stretch of an epoch on a friendster-shaped graph (an eighth of its size): 16 mini-batches in flight in turn
        dict(name="np_epoch_friendster", kind="epoch", strategy="np", nodes=8_201_045, edges=225_000_000,
             undirected=True, dim=256, dtype="bf16", cached=0.4, batch=2048, fanouts="20,15", steps=16),
        # data-parallel sampling, every hop on this GPU, operator by operator
        dict(small, name="dp_batch_small", kind="batch", strategy="dp", batch=1024, fanouts="25,10"),
        # source-split sampling for a GAT model, three hops
        dict(small, name="snp_gat_batch", kind="batch", strategy="snp_gat", batch=1024, fanouts="15,10,5"),
        # source-split sampling with virtual nodes (GraphSAGE), the short last batch of an epoch
        dict(small, name="snp_sage_batch", kind="batch", strategy="snp_sage", batch=931, fanouts="25,10"),
        # the feature stress test: 2 KiB rows, all of them cached, as many as 8 ranks exchange per step
        dict(name="gather_stress", kind="gather", rows=495_616, table=4_000_000, dim=1024, dtype="f16", missing=0.0),
        # a small gather of rows that are no multiple of a cache line, a tenth of them from host memory
        dict(name="gather_ragged", kind="gather", rows=1_203, table=200_000, dim=100, dtype="f32", missing=0.1),
        # the aggregation of the outermost papers-shaped block, hidden size 256
        dict(name="sage_papers", kind="sage", dst=67_584, fanout=15, src=151_552, dim=256, dtype="f32", segments=1),
        # column slices of four ranks' blocks in one call (feature dimension partitioned over four GPUs)
        dict(name="sage_slices", kind="sage", dst=4_099, fanout=10, src=30_011, dim=32, dtype="bf16", segments=4),
        # the attention layer of the papers-shaped configuration: 4 heads of 64
        dict(name="gat_papers", kind="gat", dst=67_584, fanout=15, src=151_552, heads=4, head_dim=64, dtype="bf16"),
        # attention from the separate operators on an inner block
        dict(name="edges_inner", kind="edges", dst=6_131, fanout=10, src=55_001, heads=4, head_dim=16, dtype="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["batch", "batch", "batch", "epoch", "gather", "gather", "sage", "sage", "gat", "gat", "edges"])
    dtype = rng.choice(["f32", "bf16", "f16"])
    if kind in ("batch", "epoch"):
        strategy = rng.choice(["np", "dp", "snp_gat", "snp_sage"]) if kind == "batch" else "np"
        nodes = _log(rng, 1 << 15, 111_000_000 if kind == "batch" else 8_200_000)
        batch = _log(rng, 100, 2048)
        # as many hops and neighbours as keep the widest hop at the listed mini-batches' size
        fanouts = [rng.randint(4, 25)]
        while len(fanouts) < 3 and rng.random() < 0.8:
            fanouts.append(rng.randint(3, 12))
        while batch * math.prod(1 + f for f in fanouts) > 1_000_000:
            fanouts = [max(2, f - 1) for f in fanouts]
        dim = _log(rng, 16, 256)
        case = dict(kind=kind, strategy=strategy, nodes=nodes, edges=int(nodes * rng.uniform(8, 14)), undirected=False,
                    dim=dim, dtype=dtype, cached=round(min(rng.uniform(0.2, 0.6), _CACHE_BYTES / (nodes * dim * _BYTES[dtype])), 3),
                    batch=batch, fanouts=",".join(map(str, fanouts)))
        if kind == "epoch":
            case["steps"] = rng.randint(6, 16)
        return case
    if kind == "gather":
        dim = _log(rng, 16, 1024)
        row = dim * _BYTES[dtype]
        missing = rng.choice([0.0, 0.0, 0.02, 0.1])
        rows = _log(rng, 500, min(495_616, (1 << 30) // row) if missing == 0.0 else 50_000)
        return dict(kind=kind, rows=rows, table=min(4_000_000, 8 * 10 ** 9 // row, rows * rng.randint(4, 200)), dim=dim, dtype=dtype,
                    missing=missing)
    dst, fanout = _log(rng, 300, 67_584), rng.randint(3, 25)
    while dst * fanout > 1_000_000:
        fanout -= 1
    src = dst + int(dst * fanout * rng.uniform(0.08, 0.9))
    if kind == "sage":
        return dict(kind=kind, dst=dst, fanout=fanout, src=src, dim=_log(rng, 4, 256), dtype=dtype,
                    segments=rng.choice([1, 1, 2, 4, 8]))
    heads = rng.choice([1, 2, 4, 8])
    head_dim = rng.choice([8, 16, 32, 64, 10, 47])
    while heads * head_dim > (256 if kind == "gat" else 64):
        heads, head_dim = (heads // 2, head_dim) if heads > 1 else (heads, head_dim // 2)
    if kind == "edges":
        while dst * fanout > 250_000:
            dst //= 2
        src = dst + int(dst * fanout * rng.uniform(0.08, 0.9))
    return dict(kind=kind, dst=dst, fanout=fanout, src=src, heads=heads, head_dim=head_dim, dtype=dtype)


# ------------------------------------------------------------------------------------------------------- data sets
class _DataSet:
    """What a training run has installed: the graph and feature tables, and the samplers made on them."""

    def __init__(self, key):
        self.key = key
        self.samplers = {}
        self.train_ids = None
        self.keep = None


_INSTALLED = None


def _install(case):
    """The case's data set, installed in the process-wide state unless it is the one installed already."""
    global _INSTALLED
    if case["kind"] == "gather":
        key = ("gather",) + tuple(case[k] for k in ("table", "dim", "dtype", "missing"))
    else:
        key = ("graph",) + tuple(case[k] for k in ("nodes", "edges", "undirected", "dim", "dtype", "cached"))
    if _INSTALLED is not None and _INSTALLED.key == key:
        return _INSTALLED
    _INSTALLED = None
    data = _DataSet(key)
    if case["kind"] == "gather":
        # nodes [0, table) are cached on the device, the nodes behind them are in host memory
        dev = torch.device("cuda", torch.cuda.current_device())
        gen = torch.Generator(device=dev).manual_seed(7)
        n_host = max(1, int(case["table"] * 0.02) if case["missing"] == 0.0 else case["table"] // 4)
        n_host = min(n_host, max(1, _HOST_BYTES // (case["dim"] * _BYTES[case["dtype"]])))
        cached = torch.empty((case["table"], case["dim"]), dtype=_TORCH[case["dtype"]], device=dev).normal_(generator=gen)
        host = torch.empty((n_host, case["dim"]), dtype=_TORCH[case["dtype"]], device=dev).normal_(generator=gen)
        ops.cache_feats_shared(case["table"] + n_host, host.cpu().pin_memory(), cached, torch.arange(case["table"]),
                               torch.arange(case["table"], case["table"] + n_host), 0)
        data.keep = n_host
    else:
        row = case["dim"] * _BYTES[case["dtype"]]
        host_rows = _HOST_BYTES // row
        w = synthetic.Workload("case", case["nodes"], case["edges"], case["dim"], case["dtype"], case["cached"],
                               _fanouts(case), 1, 256, max(0.011, min(0.5, 40_000 / case["nodes"])),
                               undirected=case["undirected"],
                               host_rows_cap=host_rows if host_rows < case["nodes"] else None)
        data.keep = synthetic.install(w)
        data.train_ids = data.keep.train_ids
    _INSTALLED = data
    return data


def _fanouts(case):
    return [int(f) for f in case["fanouts"].split(",")]


def _sampler(data, case):
    key = (case["strategy"], case["fanouts"])
    if key not in data.samplers:
        make = {"np": sampler.MixedNeighborSampler, "dp": sampler.DPNeighborSampler, "snp_gat": sampler.SPGATSampler,
                "snp_sage": sampler.SPVirtualSampler}[case["strategy"]]
        data.samplers[key] = make(0, _fanouts(case))
    return data.samplers[key]


# ------------------------------------------------------------------------------------------------- inputs of a pass
def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    if case["kind"] in ("batch", "epoch"):
        data = _install(case)
        # the draws of a pass follow from this key and the number of sampling calls made since
        ops.set_sampling(key=_SAMPLE_KEY, call_id=0)
        ids, count = data.train_ids, case.get("steps", 1)
        seeds = [ids[torch.randperm(ids.numel(), generator=gen, device=dev)[:case["batch"]]] for _ in range(count)]
        state = dict(kind=case["kind"], strategy=case["strategy"], sampler=_sampler(data, case), seeds=seeds[0])
        if case["kind"] == "epoch":
            state["batches"] = [s.cpu().pin_memory() for s in seeds]
        return state
    if case["kind"] == "gather":
        n_host = _install(case).keep
        n_miss = min(n_host, int(case["rows"] * case["missing"]))
        # a relabelled layer's input nodes: every id once, in no order
        ids = torch.cat([torch.randperm(case["table"], generator=gen, device=dev)[:case["rows"] - n_miss],
                         case["table"] + torch.randperm(n_host, generator=gen, device=dev)[:n_miss]])
        return dict(kind="gather", ids=ids[torch.randperm(ids.numel(), generator=gen, device=dev)])
    return _layer_inputs(case, gen, dev)


def _split(total, parts):
    return [total // parts + (1 if k < total % parts else 0) for k in range(parts)]


def _layer_inputs(case, gen, dev):
    """A block (or one per segment) as the samplers hand it out: `fanout` edges per destination, grouped by destination,
    sources in order of first occurrence, so that the nodes many edges share tend to come early."""
    parts = case.get("segments", 1)
    dst, src = _split(case["dst"], parts), _split(case["src"], parts)
    rows, cols = [], []
    for d, s in zip(dst, src):
        u = torch.rand(d * case["fanout"], generator=gen, device=dev, dtype=torch.float64)
        rows.append((u * u * s).long().clamp_(max=s - 1))
        cols.append(torch.arange(d, device=dev).repeat_interleave(case["fanout"]))

    def offsets(sizes):
        return torch.tensor([0] + sizes, device=dev).cumsum(0)

    def normal(*shape):
        return torch.empty(shape, dtype=_TORCH[case["dtype"]], device=dev).normal_(generator=gen)

    state = dict(kind=case["kind"], row=torch.cat(rows), col=torch.cat(cols), edges=offsets([d * case["fanout"] for d in dst]),
                 src=offsets(src), dst=offsets(dst), num_dst=case["dst"])
    if case["kind"] == "sage":
        state.update(x=normal(case["src"], case["dim"]), g=normal(case["dst"], case["dim"]))
        return state
    h, d = case["heads"], case["head_dim"]
    if case["kind"] == "gat":
        state.update(ft=normal(case["src"], h, d).requires_grad_(), el=normal(case["src"], h, 1).requires_grad_(),
                     er=normal(case["dst"], h, 1).requires_grad_(), g=normal(case["dst"], h, d))
    else:
        state.update(x=normal(case["src"], h * d), g=normal(case["dst"], h * d), el=normal(case["src"], h), er=normal(case["dst"], h))
    return state


# ------------------------------------------------------------------------------------------------------- one pass
def _sum_layer(b, x):
    off = torch.tensor([0, b.coo_row.numel(), 0, b.num_src, 0, b.num_dst]).to(x.device, non_blocking=True)
    return ops.spmm_copy_u_sum(b.coo_row, b.coo_col, x, off[0:2], off[2:4], off[4:6])


def _attention_layer(b, src, dst, heads):
    """Attention scores from a column of each head; `dst` holds the destinations' rows."""
    src, dst = src.view(src.shape[0], heads, -1), dst.view(dst.shape[0], heads, -1)
    return ops.gat_edge_softmax_sum(b.coo_row, b.coo_col, src, src[:, :, 0].contiguous(), dst[:, :, 0].contiguous(),
                                    b.num_dst)


def _forward(strategy, got):
    """The mini-batch `got` of a sampler taken through the layers: (rows of the seeds, the blocks)."""
    x = ops.load_subtensor(got[0])
    width, blocks = x.shape[1], got[2]
    if strategy == "snp_gat":
        heads = 4 if width % 4 == 0 else 1
        perm, send, recv = got[3:]
        n = blocks[0].num_dst
        src = ops.feat_shuffle(x[n:], send, recv, perm, width, 1)
        h = _attention_layer(blocks[0], src, x[:n], heads)
        for b in blocks[1:]:
            h = _attention_layer(b, h, h[:b.num_dst], heads)
        return h, blocks
    if strategy == "snp_sage":
        send, recv = got[3:]
        part = _sum_layer(blocks[0], x[blocks[1].num_dst:])
        h, rest = ops.sp_feat_shuffle(part, recv, send, int(send[1::2].sum()), width, 0), blocks[1:]
    elif strategy == "np":
        perm, send, recv, inverse = got[3:]
        h = ops.rows_gather(_sum_layer(blocks[0], x), inverse)
        h, rest = ops.feat_shuffle(h, send, recv, perm, width, 1), blocks[1:]
    else:
        h, rest = x, blocks
    for b in rest:
        h = _sum_layer(b, h)
    return h, blocks


def run(state):
    s = state
    if s["kind"] == "batch":
        got = s["sampler"].sample(None, s["seeds"])
        h, blocks = _forward(s["strategy"], got)
        # beside the result: the innermost block as it was sampled, and every block's size
        return [h, blocks[-1].coo_row, blocks[-1].coo_col] + [n for b in blocks for n in (b.num_src, b.num_dst)]
    if s["kind"] == "epoch":
        return [_forward(s["strategy"], got)[0] for got in s["sampler"].sample_iter(None, s["batches"])]
    if s["kind"] == "gather":
        return ops.load_subtensor(s["ids"])
    if s["kind"] == "sage":
        y = ops.spmm_copy_u_sum(s["row"], s["col"], s["x"], s["edges"], s["src"], s["dst"])
        gx = ops.spmm_copy_u_sum(s["col"], s["row"], s["g"], s["edges"], s["dst"], s["src"])
        return y, gx
    if s["kind"] == "gat":
        out = ops.GATEdgeSoftmaxSum.apply(s["row"], s["col"], s["ft"], s["el"], s["er"], s["num_dst"], 0.2)
        return (out,) + torch.autograd.grad(out, (s["ft"], s["el"], s["er"]), s["g"])
    score = ops.sddmm_u_add_v(s["row"], s["col"], s["el"], s["er"], s["edges"], s["src"], s["dst"])
    y = ops.spmm_u_mul_e_sum(s["row"], s["col"], s["x"], score, s["edges"], s["src"], s["dst"])
    ge = ops.sddmm_u_mul_v(s["row"], s["col"], s["x"], s["g"], s["edges"], s["src"], s["dst"])
    return score, y, ge


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _distinct(draws, nodes):
    """Expected distinct sources among `draws` edges of an R-MAT graph: a node whose id has k ones out of L bits is a
    source with probability 0.76^(L-k) 0.24^k."""
    bits = max(1, round(math.log2(nodes)))
    return sum(math.comb(bits, k) * -math.expm1(-draws * 0.76 ** (bits - k) * 0.24 ** k) for k in range(bits + 1))


def work(case):
    kind = case["kind"]
    if kind in ("batch", "epoch"):
        row = case["dim"] * _BYTES[case["dtype"]]
        total, flops, frontier = 0.0, 0.0, float(case["batch"])
        for f in reversed(_fanouts(case)):
            draws = frontier * f
            # a seed's id and its two row pointers; a drawn id read, its two block columns written; the layer's sums
            total += frontier * (24 + row) + 24 * draws
            flops += draws * case["dim"]
            frontier = min(case["nodes"], frontier + _distinct(draws, case["nodes"]))
            total += 8 * frontier
        total += frontier * (8 + 2 * row)
        steps = case.get("steps", 1)
        return {"bytes": total * steps, "flops": flops * steps}
    if kind == "gather":
        return {"bytes": case["rows"] * (16 + 2 * case["dim"] * _BYTES[case["dtype"]]), "flops": 0}
    size, edges = _BYTES[case["dtype"]], case["dst"] * case["fanout"]
    if kind == "sage":
        # each direction reads its block and one side's rows and writes the other side's
        return {"bytes": 2 * (16 * edges + (case["src"] + case["dst"]) * case["dim"] * size), "flops": 2 * edges * case["dim"]}
    width = case["heads"] * case["head_dim"]
    if kind == "gat":
        # forward: rows and scores in, sums out; backward: rows, scores and gradient in, three gradients out
        return {"bytes": 32 * edges + size * (3 * case["src"] + 2 * case["dst"]) * width + size * case["heads"] * (3 * case["src"] + 3 * case["dst"]),
                "flops": 6 * edges * width}
    return {"bytes": 48 * edges + size * (edges * (width + 2 * case["heads"]) + 2 * case["src"] * width + 2 * case["dst"] * width),
            "flops": edges * (3 * width + case["heads"])}


def tolerance(case):
    if case["kind"] == "gather":
        return "exact"          # copied rows
    if case["dtype"] == "f32":
        return {"rel": 1e-5}    # sums of 32-bit values; ids and sizes have to be the same
    return {"rel": 1e-2}        # results of 16 bits
