"""What the framework's speed is measured on: the operators and training steps that a user of
`hiscache_backend` and `hiscache` runs, from a single layer of a small batch to whole-graph blocks.

A case is a dict of plain values.  `op` names the path:

  aggr    history-aware aggregation of one block (forward, or forward + backward + admission score)
  heads   edge-weighted multi-head aggregation with gradients of rows and edge values
  cache   HistoryCache: lookup, receptive-field masks, assembly of batch.x, admission
  table   HistoryTable: per-layer lookup, masks, admission, eviction
  norm    batch norm + ReLU + dropout of a hidden layer, forward and backward
  sample  drawing one mini-batch in the fixed shape, on the device or with its sizes read by the host
  step    one training iteration (captured in a CUDA graph, or eager), SAGE or RGCN
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "history-cache_b200"))

import hiscache_backend as hb  # noqa: E402
from hiscache import HistoryCache, HistoryTrainer, HostFeatureStore, make_config  # noqa: E402
from hiscache.history_table import HistoryTable  # noqa: E402
from hiscache.sampler import Loader, SyntheticGraph  # noqa: E402

DEV = "cuda:0"
DTYPES = {"f16": torch.float16, "f32": torch.float32}
MEAN_DEGREE, EXPONENT = 14.5, 2.1       # the degree law of the headline benchmark's graph
FANOUTS = [15, 10, 5]
POOL = 16                               # batches a cache / table / step state goes round


def listed():
    return [
        # the layer next to the seeds of a 1 000-seed batch: microseconds of work, so launches and
        # host time count
        dict(name="aggr_seed_layer", op="aggr", dst=1000, deg=5, src=4500, feat=256, dtype="f32", hit=0.05,
             grad=True, skew=False),
        # first layer of a benchmark batch over raw fp16 features, which take no gradient
        dict(name="aggr_input_f16", op="aggr", dst=16500, deg=4, src=47700, feat=128, dtype="f16", hit=0.0,
             grad=False, skew=False),
        # whole-graph inference: a block far larger than the L2, fp16 rows
        dict(name="aggr_full_f16", op="aggr", dst=500000, deg=10, src=2000000, feat=128, dtype="f16", hit=0.0,
             grad=False, skew=False),
        # training on a large block with popular sources: forward, backward, admission score
        dict(name="aggr_train_f32", op="aggr", dst=200000, deg=10, src=800000, feat=256, dtype="f32", hit=0.1,
             grad=True, skew=True),
        # a width that is no multiple of four, as class counts and raw feature files have
        dict(name="aggr_odd_width", op="aggr", dst=60000, deg=12, src=200000, feat=75, dtype="f32", hit=0.05,
             grad=True, skew=False),
        # attention-style layer: weights per edge and head, both gradients
        dict(name="heads_edge_grad", op="heads", dst=100000, deg=10, src=400000, feat=64, heads=4),
        # the cache around a training step, features in pinned host memory (the history_uvm mode)
        dict(name="cache_host", op="cache", batch=1000, nodes=500000, feat=128, hidden=256, dtype="f16", host=True),
        # per-layer tables around a step, fp32 features of width 100 in HBM
        dict(name="table_layers", op="table", batch=1000, nodes=500000, feat=100, hidden=256),
        # a hidden layer's normalisation over a large batch
        dict(name="norm_large", op="norm", rows=200000, feat=256, p=0.5),
        # the loader drawing 15/10/5 neighbours for 1 000 seeds in the fixed shape
        dict(name="sample_device", op="sample", batch=1000, nodes=2000000, device=True),
        # the headline workload's step at a graph size that is quick to make
        dict(name="step_sage_captured", op="step", model="sage", captured=True, batch=1000, nodes=500000, feat=128,
             hidden=256, classes=172),
        # the heterogeneous model, eager: every batch has its own shape
        dict(name="step_rgcn_eager", op="step", model="rgcn", captured=False, batch=500, nodes=300000, feat=128,
             hidden=256, classes=153),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["aggr", "aggr", "aggr", "aggr", "heads", "cache", "table", "norm", "sample", "step"])
    if op == "aggr":
        dtype = rng.choice(["f16", "f32"])
        grad = dtype == "f32" and rng.random() < 0.7
        feat = rng.choice([64, 100, 128, 256]) if rng.random() < 0.6 else rng.randint(33, 400)
        deg = rng.randint(3, 15)
        # no more gathered bytes than the largest listed block
        most = 1.2e9 / (deg * feat * (4 if dtype == "f32" else 2)) / (2 if grad else 1)
        dst = _log_int(rng, 500, max(1000, min(500000, most)))
        return dict(op=op, dst=dst, deg=deg, src=int(dst * rng.uniform(1.5, 5)), feat=feat, dtype=dtype,
                    hit=rng.choice([0.0, 0.05, 0.25]), grad=grad, skew=rng.random() < 0.5)
    if op == "heads":
        heads, feat = rng.choice([2, 4, 8]), rng.choice([16, 32, 48, 64])
        dst = _log_int(rng, 1000, 100000 * 256 // max(256, heads * feat))
        return dict(op=op, dst=dst, deg=rng.randint(3, 10), src=int(dst * rng.uniform(1.5, 4)), feat=feat, heads=heads)
    if op == "cache":
        return dict(op=op, batch=_log_int(rng, 100, 1000), nodes=_log_int(rng, 200000, 500000),
                    feat=rng.choice([64, 128, 200]), hidden=rng.choice([128, 256]), dtype=rng.choice(["f16", "f32"]),
                    host=rng.random() < 0.5)
    if op == "table":
        return dict(op=op, batch=_log_int(rng, 100, 1000), nodes=_log_int(rng, 200000, 500000),
                    feat=rng.choice([64, 100, 128]), hidden=rng.choice([128, 256]))
    if op == "norm":
        return dict(op=op, rows=_log_int(rng, 1000, 200000), feat=rng.choice([64, 128, 172, 256]),
                    p=rng.choice([0.0, 0.5]))
    if op == "sample":
        return dict(op=op, batch=_log_int(rng, 100, 1000), nodes=_log_int(rng, 300000, 2000000),
                    device=rng.random() < 0.7)
    model = rng.choice(["sage", "sage", "rgcn"])
    batch = _log_int(rng, 100, 1000 if model == "sage" else 500)
    return dict(op="step", model=model, captured=model == "sage" and rng.random() < 0.6, batch=batch,
                nodes=_log_int(rng, 200000, 500000), feat=rng.choice([64, 128]), hidden=rng.choice([128, 256]),
                classes=rng.choice([47, 172]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _block(c, g):
    """One CSR block of dst * deg edges in ragged rows; with `skew` the sources follow the popularity
    law of the synthetic graph (floor(n * u^3)), otherwise they are uniform."""
    edges = c["dst"] * c["deg"]
    n = torch.bincount(torch.randint(0, c["dst"], (edges,), generator=g, device=DEV), minlength=c["dst"])
    ptr = torch.zeros(c["dst"] + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(n, 0, out=ptr[1:])
    if c.get("skew"):
        u = torch.rand(edges, generator=g, device=DEV, dtype=torch.float64)
        idx = (u.pow_(3.0) * c["src"]).to(torch.int64).clamp_(max=c["src"] - 1)
    else:
        idx = torch.randint(0, c["src"], (edges,), generator=g, device=DEV)
    return ptr, idx


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=DEV)


def _graph(c, seed):
    return SyntheticGraph(c["nodes"], MEAN_DEGREE, EXPONENT, c.get("classes", 47), seed=seed, device=DEV,
                          num_train=c["nodes"] // 4)


def _cache_gb(c):
    """A device cache of a seventh of the features' size, as 4 GB is of the benchmark's 28 GB."""
    return c["nodes"] * c["feat"] * (2 if c.get("dtype", "f16") == "f16" else 4) / 7 / 1024 ** 3


def _features(c, seed, dtype, host=True):
    if host:
        return HostFeatureStore.synthetic(c["nodes"], c["feat"], dtype, seed, DEV)
    return HostFeatureStore(_randn(_gen(seed), c["nodes"], c["feat"]).to(dtype), DEV)


def _caps(c, fan):
    """Rows per layer and edges of a fixed-shape batch, with room for every batch of the case."""
    nodes, edges = _batch(c, fan)
    up = lambda v: -(-int(v * 1.02 + 250) // 128) * 128  # noqa: E731
    return [c["batch"]] + [up(n) for n in nodes[1:]], up(edges[-1])


def _batches(c, loader):
    return list(loader.iterate_fixed(POOL, *_caps(c, FANOUTS), reuse=POOL))


def _embeddings(g, batches, hidden):
    """For every batch the produced rows of its first hop and the gradient that reached them."""
    n = max(int(b.num_node_in_layer[1]) for b in batches)
    rows = _randn(g, n, hidden)
    grads = [_randn(g, int(b.num_node_in_layer[1]), hidden) * 1e-3 for b in batches]
    return [(rows[:gr.shape[0]], gr) for gr in grads]


class _Round:
    """A pool of batches, gone round one per pass.  Its POOL batches are more than the ten iterations
    after which the history ring restarts, so a batch that comes back finds the history of others."""

    def __init__(self, batches):
        self.batches, self.k = batches, 0

    def next(self):
        k = self.k % len(self.batches)
        self.k += 1
        return k, self.batches[k]

    def following(self):
        return self.batches[self.k % len(self.batches)]


def prepare(case, seed):
    return {"aggr": _prepare_aggr, "heads": _prepare_heads, "cache": _prepare_cache, "table": _prepare_table,
            "norm": _prepare_norm, "sample": _prepare_sample, "step": _prepare_step}[case["op"]](case, seed)


def _prepare_aggr(c, seed):
    g = _gen(seed)
    ptr, idx = _block(c, g)
    s = {"c": c, "ptr": ptr, "idx": idx, "x": _randn(g, c["src"], c["feat"]).to(DTYPES[c["dtype"]]), "map": None,
         "table": None}
    if c["hit"] > 0:
        cap = max(64, c["dst"] // 4)
        slot = torch.randint(0, cap, (c["dst"],), generator=g, device=DEV)
        s["map"] = torch.where(torch.rand(c["dst"], generator=g, device=DEV) < c["hit"], slot, -1)
        s["table"] = _randn(g, cap, c["feat"]).to(DTYPES[c["dtype"]])
    if c["grad"]:
        s["x"].requires_grad_(True)
        s["grad"] = _randn(g, c["dst"], c["feat"])
        s["score"] = torch.empty(c["dst"], device=DEV)
    return s


def _prepare_heads(c, seed):
    g = _gen(seed)
    ptr, idx = _block(c, g)
    H, F = c["heads"], c["feat"]
    w = torch.rand((idx.shape[0], H), generator=g, device=DEV)     # attention weights are positive
    return {"c": c, "ptr": ptr, "idx": idx, "x": _randn(g, c["src"], H, F).requires_grad_(True),
            "w": w.requires_grad_(True), "grad": _randn(g, c["dst"], H, F)}


def _prepare_cache(c, seed):
    g = _gen(seed)
    graph = _graph(c, seed)
    cfg = make_config(feature_dim=c["feat"], num_classes=47, hidden_dim=c["hidden"], num_layers=3,
                      num_nodes=c["nodes"], device=DEV, limit=_cache_gb(c), batch_size=c["batch"])
    t = HistoryCache(uvm=_features(c, seed, DTYPES[c["dtype"]], c["host"]), config=cfg, mode="history_uvm",
                     total_num_node=c["nodes"], sorted_indices=graph.sorted_indices, storage_dtype=DTYPES[c["dtype"]])
    batches = _batches(c, Loader(graph, FANOUTS, c["batch"], "history_uvm", seed=seed))
    s = {"c": c, "table": t, "round": _Round(batches), "made": _embeddings(g, batches, c["hidden"]), "iter": 1}
    for _ in range(3):      # a history that is in use
        _run_cache(s)
    return s


def _prepare_table(c, seed):
    g = _gen(seed)
    graph = _graph(c, seed)
    cfg = make_config(feature_dim=c["feat"], num_classes=47, hidden_dim=c["hidden"], num_layers=3,
                      num_nodes=c["nodes"], device=DEV, batch_size=c["batch"], buffer_size=[200000, 50000])
    batches = _batches(c, Loader(graph, FANOUTS, c["batch"], "memory", seed=seed))
    made = []
    for b in batches:
        nn = [int(v) for v in b.num_node_in_layer]
        made.append([(_randn(g, nn[2], c["feat"]), _randn(g, nn[2], c["feat"]) * 1e-3),
                     (_randn(g, nn[1], c["hidden"]), _randn(g, nn[1], c["hidden"]) * 1e-3)])
    s = {"c": c, "table": HistoryTable(cfg, total_num_node=c["nodes"]), "round": _Round(batches), "made": made,
         "iter": 0}
    for _ in range(3):
        _run_table(s)
    return s


def _prepare_norm(c, seed):
    g = _gen(seed)
    n, F = c["rows"], c["feat"]
    return {"c": c, "x": (_randn(g, n, F) * 2 + 0.5).requires_grad_(True),
            "w": (1 + 0.1 * _randn(g, F)).requires_grad_(True), "b": (0.1 * _randn(g, F)).requires_grad_(True),
            "mean": torch.zeros(F, device=DEV), "var": torch.ones(F, device=DEV), "grad": _randn(g, n, F),
            "state": torch.zeros(4, dtype=torch.int64, device=DEV), "seed": int(seed)}


def _prepare_sample(c, seed):
    loader = Loader(_graph(c, seed), FANOUTS, c["batch"], "history_uvm", seed=seed)
    caps, edge_cap = _caps(c, FANOUTS)
    draw_batches = loader.iterate_fixed if c["device"] else loader.iterate_padded
    return {"c": c, "it": draw_batches(1 << 40, caps, edge_cap)}


# relation of an edge by the types of its destination and its source (three node types)
REL_TABLE = [0, 1, 2, 1, 3, 4, 2, 4, 0]


def _prepare_step(c, seed):
    torch.manual_seed(seed)
    graph = _graph(c, seed)
    sage = c["model"] == "sage"
    fan = FANOUTS if sage else [25, 15]
    cfg = make_config(feature_dim=c["feat"], num_classes=c["classes"], hidden_dim=c["hidden"], num_layers=len(fan),
                      num_nodes=c["nodes"], model=c["model"], device=DEV, limit=_cache_gb(c), batch_size=c["batch"],
                      fanouts=fan, num_rel=1 if sage else 5)
    if not sage:
        n = c["nodes"]
        cfg.dl.dataset["type_bounds"] = [0, n // 2, n - n // 100, n]
        cfg.dl.dataset["rel_table"] = REL_TABLE
    loader = Loader(graph, fan, c["batch"], "history_uvm", seed=seed)
    t = HistoryTrainer(cfg, graph=graph, uvm=_features(c, seed, torch.float16), loader=loader,
                       storage_dtype=torch.float16, seed=seed)
    t.model.train()
    for k, bn in enumerate(t.model.bns):        # dropout of this state depends on its seed alone
        bn.drop_seed = int(seed) * 16 + k
    if c["captured"]:
        batches = _batches(c, loader)
        t.enable_cuda_graph(*_caps(c, fan), batches[:2])
    else:
        batches = list(loader._iterate(POOL))
    s = {"c": c, "trainer": t, "round": _Round(batches)}
    for _ in range(2):
        _run_step(s)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    return {"aggr": _run_aggr, "heads": _run_heads, "cache": _run_cache, "table": _run_table, "norm": _run_norm,
            "sample": _run_sample, "step": _run_step}[state["c"]["op"]](state)


def _run_aggr(s):
    c = s["c"]
    if not c["grad"]:
        return hb.aggr_forward(s["x"], s["ptr"], s["idx"], c["dst"], history_map=s["map"], history_buffer=s["table"],
                               indexed=True, force_grad=False)
    out = hb.aggr_forward(s["x"], s["ptr"], s["idx"], c["dst"], history_map=s["map"], history_buffer=s["table"],
                          indexed=True, score_out=hb.ScoreSink(s["score"]))
    gx, = torch.autograd.grad(out, s["x"], s["grad"])
    return out.detach(), gx, s["score"]


def _run_heads(s):
    out = hb.aggr_forward_history_edge_value(s["x"], s["ptr"], s["idx"], s["w"], None, None, 0, s["c"]["dst"])
    gx, gw = torch.autograd.grad(out, (s["x"], s["w"]), s["grad"])
    return out.detach(), gx, gw


def _run_cache(s):
    t = s["table"]
    k, b = s["round"].next()
    t.lookup_and_load(b)
    rows, grad = s["made"][k]
    rows = rows.detach()
    rows.grad = grad                     # what the model's backward pass leaves behind
    t.produced_embedding = rows
    t.update_history(b, s["iter"])
    s["iter"] += 1
    return {"x": b.x, "sub2embed": t.sub2embed, "sub2feat": t.sub2feat, "used": t.used_masks, "map": t.full2embed,
            "ring": t.embed2full, "buffer": t.buffer, "header": t._header}


class _Grad:
    """An aggregation output with its gradient, as a conv leaves it in `history_out`."""

    def __init__(self, rows, grad):
        self.rows, self.grad = rows, grad

    def __getitem__(self, k):
        return self.rows[k]


def _run_table(s):
    t = s["table"]
    k, b = s["round"].next()
    nn = b.num_node_in_layer
    t.lookup(b.sub_to_full, nn)
    used = hb.count_history_reconstruct(b.ptr, b.idx, t.sub_to_history[1], b.sub_to_full.shape[0], b.y.shape[0], 3)
    t.history_out = [_Grad(rows, grad) for rows, grad in s["made"][k]]
    t.record_history(b.sub_to_full, b, s["iter"], used)
    t.evict_history(b, s["iter"])
    s["iter"] += 1
    return {"hits": t.sub_to_history, "used": used, "slots": t.full_to_history_layered,
            "nodes": t.history_to_full_layered, "checkin": t.checkin_iter, "rows": t.history_buffer_layered,
            "header": t.cuda_header_layered}


def _run_norm(s):
    y = hb.norm_act(s["x"], s["w"], s["b"], s["state"], running_mean=s["mean"], running_var=s["var"], p=s["c"]["p"],
                    seed=s["seed"])
    gx, gw, gb = torch.autograd.grad(y, (s["x"], s["w"], s["b"]), s["grad"])
    return y.detach(), gx, gw, gb, s["mean"], s["var"]


def _run_sample(s):
    b = next(s["it"])
    return {"ptr": b.ptr, "idx": b.idx, "nodes": b.sub_to_full, "y": b.y, "mask": b.mask}


def _run_step(s):
    t, r = s["trainer"], s["round"]
    _, b = r.next()
    loss = t.train_step(b, r.following() if s["c"]["captured"] else None)
    # a bias in front of a batch norm has no gradient but rounding noise, which Adam turns into
    # steps of full length: it changes no result and is left out
    w = {k: p.detach() for k, p in t.model.named_parameters() if "lin_l.bias" not in k}
    h = t.table
    return {"loss": loss.detach(), "weights": w, "map": h.full2embed, "ring": h.embed2full, "buffer": h.buffer,
            "header": h._header}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _distinct(c):
    """Expected number of distinct sources among the block's edges."""
    e = c["dst"] * c["deg"] / c["src"]
    if not c.get("skew"):
        return c["src"] * (1 - math.exp(-e))
    x = (np.arange(20000) + 0.5) / 20000        # popularity density of floor(n * u^3)
    return c["src"] * float(np.mean(1 - np.exp(-e * x ** (-2 / 3) / 3)))


def _batch(c, fan):
    """Expected rows per layer and edges of a sampled batch, from the graph's degree law."""
    u = (np.arange(20000) + 0.5) / 20000
    raw = np.minimum(u ** (-1 / (EXPONENT - 1)), 1e5)
    deg = np.maximum(np.floor(raw * MEAN_DEGREE / raw.mean()), 1)
    nodes, edges, frontier = [c["batch"]], [], c["batch"]
    for f in fan:
        e = frontier * float(np.minimum(deg, f).mean())
        frontier = 0.68 * e                      # the rest are nodes that the batch has already
        edges.append((edges[-1] if edges else 0) + e)
        nodes.append(nodes[-1] + frontier)
    return nodes, edges


def work(case):
    c, op = case, case["op"]
    if op in ("aggr", "heads"):
        n, e, width = c["dst"], c["dst"] * c["deg"], c["feat"] * c.get("heads", 1)
        size = 2 if c.get("dtype") == "f16" else 4
        miss = 1 - c.get("hit", 0.0)
        b = miss * _distinct(c) * width * size + (1 - miss) * n * width * size + n * width * 4 + 8 * (n + 1 + e)
        b += 8 * n if miss < 1 else 0
        flops = miss * e * width
        if op == "heads":
            b += n * width * 4 + c["src"] * width * 4 + 2 * 4 * e * c["heads"]
            flops *= 6
        elif c["grad"]:
            b += n * width * 4 + c["src"] * width * 4 + 4 * n
            flops = 2 * flops + 2 * n * width
        return {"bytes": b, "flops": flops}
    if op == "norm":
        # x and grad_y in, y and grad_x out
        return {"bytes": 4 * c["rows"] * c["feat"] * 4, "flops": 20 * c["rows"] * c["feat"]}
    fan = [25, 15] if c.get("model") == "rgcn" else FANOUTS
    nodes, edges = _batch(c, fan)
    if op == "sample":
        # per frontier row two ptr entries, per draw one neighbour; the batch's arrays out
        return {"bytes": 24 * nodes[-2] + 16 * edges[-1] + 17 * nodes[-1] + 16 * c["batch"], "flops": 10 * edges[-1]}
    csr = 8 * (nodes[-2] + edges[-1])
    size = 4 if c.get("dtype") == "f32" else 2
    if op == "cache":
        # ids, two map reads, rows in and out; scores; the lower half of the candidates admitted
        adm = nodes[1] / 2
        b = csr + nodes[-1] * (8 + 2 * 8 + 2 * c["feat"] * size + 4) + nodes[1] * (8 + 4 * c["hidden"])
        return {"bytes": b + adm * (c["hidden"] * (4 + size) + 24), "flops": 2 * nodes[1] * c["hidden"]}
    if op == "table":
        b = csr + 4 * nodes[-1] + 8 * (200000 + 50000)       # the check-in times are looked through for stale rows
        for n, width in ((nodes[2], c["feat"]), (nodes[1], c["hidden"])):
            b += n * (8 + 2 * 8 + 4 * width) + n / 2 * (2 * 4 * width + 24)
        return {"bytes": b, "flops": 2 * (nodes[2] * c["feat"] + nodes[1] * c["hidden"])}
    # step: feature rows in, activations and their gradients once each, weights and Adam's state
    widths = [c["feat"]] + [c["hidden"]] * (len(fan) - 1) + [c["classes"]]
    b, flops = csr + nodes[-1] * (24 + c["feat"] * 2), 0
    per = 2 if c["model"] == "sage" else 5
    for k in range(len(fan)):
        n, w_in, w_out = nodes[len(fan) - 1 - k], widths[k], widths[k + 1]
        b += n * (w_in + 2 * w_out) * 4 + 7 * 4 * per * w_in * w_out
        flops += (2 if k == 0 else 3) * 2 * per * n * w_in * w_out
    return {"bytes": b, "flops": flops}


def tolerance(case):
    if case["op"] in ("cache", "table", "sample"):
        return "exact"          # maps, masks, row copies and a threshold of fixed arithmetic
    if case["op"] == "step":
        # fp32 products and sums in other orders, one Adam step on top of them; a score next to the
        # threshold may fall on its other side
        return {"rel": 1e-4, "max": 2e-2, "differ": 1e-3}
    return {"rel": 1e-5, "max": 1e-3}
