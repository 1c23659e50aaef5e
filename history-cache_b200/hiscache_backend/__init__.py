"""`hiscache_backend`: the operator module of HisCache, backed by libhiscache_b200.

The eight functions of the reference's pybind11 module keep their names,
argument order and meaning (src/cpp/python_bindings/binding.cpp:9-19):

    record_history, count_history_reconstruct, count_num,
    get_graph_structure_score, aggr_forward_history,
    aggr_forward_history_edge_value, p2psend, p2psend_gentensor

Differences that a caller can observe: argument errors raise RuntimeError
instead of ending the process (src/cpp/include/common.h:13-34); ring slots in
record_history follow ascending row order instead of warp-scheduling order
(src/cpp/src/grad_check.cu:25); history_size == 0 means "no history" instead
of exit(1) (src/cpp/src/history_aggr.cu:440-441).

The functions below the line are the wider operators the `hiscache` package
uses: history rows read straight from the table, per-source select inside the
gather, fp16 storage, the admission score fused into the backward pass, the
device-side threshold and admission, row assembly from host-resident features.
"""
from __future__ import annotations

import ctypes as C
import os

import torch

from . import _capi
from . import _native
from ._capi import (HC_F16, HC_F32, HC_SCORE_L1, HC_SCORE_L2, AggrArgs, check, dtype_code, i64c,
                    lib, on_device, ptr, require_cuda, rows2d, scratch, stream_of)

__all__ = [
    "record_history", "count_history_reconstruct", "count_num", "get_graph_structure_score",
    "aggr_forward_history", "aggr_forward_history_edge_value", "p2psend", "p2psend_gentensor",
    "aggr_forward", "score_rows", "record_history_noalloc", "select_threshold", "cache_admit", "evict_stale",
    "evict_by_score", "evict_stale_dev", "stamp_checkin", "CHECKIN_MARKER", "map_lookup", "gather_rows", "load_rows", "bucket_by_owner",
    "unpermute_rows", "owner_lookup", "bucket_pad", "unpad_hits", "last_occurrence", "sample_hop", "relabel", "relabel_seed",
    "relabel_reset", "mix64", "cache_lookup", "evict_both", "launch_count", "ScoreSink", "KernelTimer",
    "set_kernel_timer", "prepare_aggr", "run_aggr_fwd", "run_aggr_bwd", "transpose_block", "run_aggr_bwd_gather",
    "PeerRegion", "peer_open", "peer_close", "peer_ptrs", "peer_lookup", "peer_publish", "peer_pull", "peer_admit", "make_shard",
]

def launch_count() -> int:
    """Number of kernels of this library launched so far in this process."""
    return _native.launches()


_called = _native.add_launches


class KernelTimer:
    """Collects CUDA-event pairs around library calls (set with set_kernel_timer).
    `only`: record just the calls whose tag starts with this prefix."""

    def __init__(self, only=None):
        self.records = []
        self.only = only

    def summary(self):
        torch.cuda.synchronize()
        agg = {}
        for name, e0, e1 in self.records:
            a = agg.setdefault(name, {"launches": 0, "ms_total": 0.0})
            a["launches"] += 1
            a["ms_total"] += e0.elapsed_time(e1)
        return agg


_timer = None


def set_kernel_timer(t):
    """While a KernelTimer is set, every library call is bracketed by two CUDA events on the
    stream it launches on."""
    global _timer
    _timer = t
    _native.set_timed(t is not None)


class _span:
    __slots__ = ("name", "dev", "e0")

    def __init__(self, name, dev):
        self.name, self.dev, self.e0 = name, dev, None

    def __enter__(self):
        if _timer is not None and (_timer.only is None or self.name.startswith(_timer.only)):
            self.e0 = torch.cuda.Event(enable_timing=True)
            self.e0.record(torch.cuda.current_stream(self.dev))
        return self

    def __exit__(self, *exc):
        if self.e0 is not None:
            e1 = torch.cuda.Event(enable_timing=True)
            e1.record(torch.cuda.current_stream(self.dev))
            _timer.records.append((self.name, self.e0, e1))
        return False


_native.open_library(_capi.lib._handle)
_native.set_span(_span)


def _tag(name, t):
    return f"{name}[{'f16' if t.dtype == torch.float16 else 'f32'},F={t.shape[-1]}]"


ScoreSink = _native.ScoreSink


def _empty(t):
    return t is None or (isinstance(t, torch.Tensor) and t.numel() == 0)


# ---------------------------------------------------------------------------
# aggregation
# ---------------------------------------------------------------------------
def _aggr_args(inp, ptr_t, idx_t, num_node, edge_value, hmap, hbuf, h_indexed, src_map, src_alt):
    a = AggrArgs()
    a.struct_size = C.sizeof(AggrArgs)
    multi = inp.dim() == 3
    H = inp.shape[1] if multi else 1
    F = inp.shape[-1]
    a.ptr, a.idx, a.num_node = ptr(ptr_t), ptr(idx_t), num_node
    a.input, a.in_dtype, a.feat, a.num_head = ptr(inp), dtype_code(inp), F, H
    a.n_src, a.in_stride = inp.shape[0], inp.stride(0) if inp.shape[0] > 1 else H * F
    if src_map is not None:
        a.src_map, a.src_alt = ptr(src_map), ptr(src_alt)
        a.alt_dtype = dtype_code(src_alt)
        a.alt_stride = src_alt.stride(0) if src_alt.shape[0] > 1 else H * F
        a.alt_rows = src_alt.shape[0]
    a.edge_value = ptr(edge_value)
    if hmap is not None:
        a.hmap, a.hbuf, a.h_dtype = ptr(hmap), ptr(hbuf), dtype_code(hbuf)
        a.h_indexed = 1 if h_indexed else 0
        a.hsize = hbuf.stride(0) if hbuf.dim() > 1 and hbuf.shape[0] > 1 else hbuf.shape[-1]
        a.h_rows = hbuf.shape[0] if hbuf.dim() > 1 else 1
    return a


def aggr_forward(input, ptr, idx, num_node=0, *, history_map=None, history_buffer=None,
                 indexed=False, edge_value=None, src_map=None, src_alt=None, score_out=None,
                 score_kind=HC_SCORE_L2, force_grad=True):
    """History-aware aggregation.

    out[r] = history row if history_map[r] != -1 else mean (or edge-weighted sum) of the
    source rows of r's neighbours.  `indexed=True` reads row history_map[r] of
    `history_buffer` (the table itself); otherwise row r (a row-aligned gather, the
    reference layout).  `src_map`/`src_alt` choose, per source, a cached row instead of the
    fresh one.  If `score_out` (fp32 [num_node], or a ScoreSink holding one) is given, the
    backward pass writes the per-row admission score of the incoming gradient into it.
    With force_grad (the default) the result requires grad even when no input does
    (history_aggr.cu:604), which is what lets a caller retain_grad() it.
    """
    return _native.aggr(input, ptr, idx, int(num_node), history_map, history_buffer, indexed, edge_value, src_map,
                        src_alt, score_out, score_kind, force_grad, DETERMINISTIC_BWD, GATHER_MIN_BYTES,
                        GATHER_MIN_FEAT)


class PreparedAggr:
    """A filled hc_aggr_args plus references that keep its tensors alive."""

    def __init__(self, args, keep, dev, tag):
        self.args, self.keep, self.dev, self.tag = args, keep, dev, tag


def prepare_aggr(input, ptr, idx, num_node, *, history_map=None, history_buffer=None,
                 indexed=False, edge_value=None, src_map=None, src_alt=None):
    """Descriptor for run_aggr_fwd / run_aggr_bwd: the operators without autograd."""
    dev = require_cuda(input, ptr, idx, edge_value, history_map, history_buffer, src_map, src_alt)
    a = _aggr_args(input, ptr, idx, int(num_node), edge_value, history_map, history_buffer, indexed,
                   src_map, src_alt)
    return PreparedAggr(a, (input, ptr, idx, edge_value, history_map, history_buffer, src_map, src_alt),
                        dev, _tag("", input))


def run_aggr_fwd(p: PreparedAggr, out):
    with torch.cuda.device(p.dev), _span("hc_aggr_fwd" + p.tag, p.dev):
        check(lib.hc_aggr_fwd(C.byref(p.args), ptr(out), stream_of(p.dev)), "hc_aggr_fwd")
    _called()
    return out


def run_aggr_bwd(p: PreparedAggr, grad_out, grad_input=None, grad_history=None, edge_grad=None,
                 score=None, score_kind=HC_SCORE_L2, zero=True):
    with torch.cuda.device(p.dev), _span("hc_aggr_bwd" + p.tag, p.dev):
        check(lib.hc_aggr_bwd(C.byref(p.args), ptr(grad_out), ptr(grad_input), 1 if zero else 0,
                              ptr(grad_history), ptr(edge_grad), ptr(score), score_kind,
                              stream_of(p.dev)), "hc_aggr_bwd")
    _called()


# The scatter is bound by read-modify-write DRAM traffic once grad_input no longer fits the 126 MB L2;
# below that its lines stay in L2 and it needs fewer launches.  Blocks whose grad_input is at least this
# large, in rows of at least GATHER_MIN_FEAT columns, take the backward by source (hc_aggr_bwd_source).
# Measured on B200, forward + backward of uniform blocks of 10 edges a row, three sources to a
# destination, scatter against by source: 1 KB rows, 98 MB of gradient 123 / 124 us, 197 MB 295 / 223 us,
# 393 MB 650 / 467 us; 512 B rows, 197 MB 311 / 281 us; 256 B rows, 98 MB 150 / 218 us; 4 heads of 64 with
# the gradient of the weights, 98 MB 199 / 191 us, 307 MB 644 / 472 us.
GATHER_MIN_BYTES = int(os.environ.get("HISCACHE_BWD_GATHER_MIN_BYTES", 128 << 20))
GATHER_MIN_FEAT = int(os.environ.get("HISCACHE_BWD_GATHER_MIN_FEAT", 128))


# True: every aggregation backward that can takes the transposed gather, whose sums have a fixed
# order, so a training step is reproducible bit for bit (the scatter's atomics are not)
DETERMINISTIC_BWD = os.environ.get("HISCACHE_DETERMINISTIC_BWD", "0") not in ("", "0")


def transpose_block(p: PreparedAggr, max_edges):
    """(t_ptr [n_src+1], t_dst [max_edges], t_w [max_edges]): per source the ascending list of
    miss destination rows that have it as a neighbour, with the weight 1/deg of each."""
    dev, a = p.dev, p.args
    n_src = int(a.n_src)
    n_edges = max(int(max_edges), 1)
    t_ptr = torch.empty(n_src + 1, dtype=torch.int64, device=dev)
    t_dst = torch.empty(n_edges, dtype=torch.int64, device=dev)
    t_w = torch.empty(n_edges, dtype=torch.float32, device=dev)
    sc = scratch(dev, lib.hc_transpose_scratch_bytes(n_src, n_edges), "transpose")
    with on_device(dev), _span("hc_transpose_block", dev):
        check(lib.hc_transpose_block(C.byref(a), int(max_edges), ptr(t_ptr), ptr(t_dst), ptr(t_w), ptr(sc),
                                     stream_of(dev)), "hc_transpose_block")
    _called(2 + 5 * max(1, (max(n_src, 1).bit_length() + 7) // 8))
    return t_ptr, t_dst, t_w


def declare_batch(ptr_t, idx_t, n_nodes):
    """Tells the library that (ptr, idx) is the CSR of one sampled batch over `n_nodes` local ids
    that all layers aggregate over (layer k uses the rows [0, num_node_k)).  The backward passes
    of the batch can then share ONE transposition (see shared_transpose)."""
    _native.declare_batch(ptr_t, idx_t, int(n_nodes))


def shared_transpose(ptr_t, idx_t):
    """(t_ptr, t_dst, t_w, n_edges) of a declared batch's whole CSR, built once and reused by the
    backward pass of every layer: all layers aggregate over a prefix of the same (ptr, idx), and a
    source's list is sorted by destination row, so the list of a smaller layer is a prefix of it
    (hc_aggr_bwd_gather skips the rest).  None when (ptr, idx) was not declared."""
    return _native.shared_transpose(ptr_t, idx_t)


def run_aggr_bwd_gather(p: PreparedAggr, t_ptr, t_dst, t_w, grad_out, grad_input, n_edges=None):
    n_edges = int(t_dst.shape[0] if n_edges is None else n_edges)
    feat = int(p.args.feat)
    sc = scratch(p.dev, lib.hc_gather_scratch_bytes(n_edges, feat), "gather") if n_edges > 64 else None
    with torch.cuda.device(p.dev), _span("hc_aggr_bwd_gather" + p.tag, p.dev):
        check(lib.hc_aggr_bwd_gather(C.byref(p.args), ptr(t_ptr), ptr(t_dst), ptr(t_w), t_ptr.shape[0] - 1,
                                     n_edges, ptr(grad_out), ptr(grad_input), ptr(sc), stream_of(p.dev)),
              "hc_aggr_bwd_gather")
    _called(4 if n_edges > 64 else 1)


def aggr_forward_history(input, ptr, idx, history_map, history_buffer, history_size, num_node):
    """src/cpp/src/history_aggr.cu:598-606.  history_buffer is row-aligned: row r of it
    replaces output row r where history_map[r] != -1."""
    if history_size == 0:
        history_map = history_buffer = None
    elif not _empty(history_buffer) and history_buffer.dim() == 1:
        history_buffer = history_buffer.view(-1, history_size)
    return aggr_forward(input, ptr, idx, num_node, history_map=history_map,
                        history_buffer=history_buffer)


def aggr_forward_history_edge_value(input, ptr, idx, edge_value, history_map, history_buffer,
                                    history_size, num_node):
    """src/cpp/src/history_aggr.cu:608-617: weighted sum; edge_value [E] or [E, H] with
    input [n, H, F]."""
    if history_size == 0:
        history_map = history_buffer = None
    elif not _empty(history_buffer) and history_buffer.dim() == 1:
        history_buffer = history_buffer.view(-1, history_size)
    if _empty(edge_value):
        raise RuntimeError("aggr_forward_history_edge_value: edge_value is empty")
    if edge_value.dim() == 2 and (input.dim() != 3 or input.shape[1] != edge_value.shape[1]):
        raise RuntimeError("multi-head edge_value needs input [n, num_head, feat] "
                           "(history_aggr.cu:421-422)")
    return aggr_forward(input, ptr, idx, num_node, history_map=history_map,
                        history_buffer=history_buffer, edge_value=edge_value)


# ---------------------------------------------------------------------------
# batch norm + ReLU + dropout in one forward pair / one backward pair
# ---------------------------------------------------------------------------
def norm_act(x, weight, bias, state, *, valid=None, running_mean=None, running_var=None, momentum=0.1,
             eps=1e-5, p=0.0, relu=True, seed=0, num_batches_tracked=None):
    """y = dropout(relu(batch_norm(x))) with batch statistics (training mode), as two kernels
    forward and two backward (csrc/norm_act.cu).  `state`: int64[4] CUDA tensor, zero-initialised
    once and private to the calling layer (dropout step counter).  `valid`: optional row mask.
    `num_batches_tracked`: BatchNorm1d's counter, advanced by the same kernel."""
    return _native.norm_act(x, weight, bias, state, valid, running_mean, running_var, momentum, eps, p, relu,
                            seed & 0xFFFFFFFFFFFFFFFF, num_batches_tracked)


def norm_act_supported(x) -> bool:
    return x.is_cuda and x.dtype == torch.float32 and x.dim() == 2 and x.shape[1] % 4 == 0 and x.shape[1] <= 1024


# ---------------------------------------------------------------------------
# scores, threshold, admission, eviction (csrc/torch_ops.cpp)
# ---------------------------------------------------------------------------
score_rows = _native.score_rows
select_threshold = _native.select_threshold
record_history = _native.record_history
cache_admit = _native.cache_admit
evict_stale = _native.evict_stale
evict_stale_dev = _native.evict_stale_dev
evict_by_score = _native.evict_by_score
evict_both = _native.evict_both
stamp_checkin = _native.stamp_checkin


def record_history_noalloc(buffer_new, buffer_all, used_mask, sub_to_full, sub_to_history,
                           history_to_full, full_to_history, header, score, thres, checkin_iter,
                           glb_iter, n_admitted=None):
    """record_history through the entry point that carries its own scratch
    (hc_record_history_noalloc): for hosts that cannot allocate device memory themselves.
    This wrapper allocates nothing either; every argument must already be a contiguous CUDA
    tensor of the right dtype (fp32 rows / scores / thres, int64 maps, bool mask).  At most
    hc_noalloc_max_rows() candidate rows; calls on one device must not overlap on the GPU."""
    dev = require_cuda(buffer_new, buffer_all, sub_to_full, sub_to_history, history_to_full,
                       full_to_history, header, score, thres, checkin_iter)
    n, hs = buffer_new.shape
    for t in (buffer_new, buffer_all, sub_to_full, sub_to_history, history_to_full, full_to_history,
              header, score, thres, checkin_iter):
        if not t.is_contiguous():
            raise RuntimeError("record_history_noalloc: arguments must be contiguous")
    if buffer_new.dtype != torch.float32 or score.dtype != torch.float32 or thres.dtype != torch.float32:
        raise TypeError("record_history_noalloc: rows, score and thres must be float32")
    # the same argument checks as record_history (comparisons only, nothing is allocated):
    # a narrower table or 32-bit maps would otherwise be read out of bounds on the device
    if buffer_all.dim() != 2 or buffer_all.shape[1] != hs:
        raise RuntimeError("record_history_noalloc: row widths differ")
    for name, t in (("sub_to_full", sub_to_full), ("sub_to_history", sub_to_history),
                    ("history_to_full", history_to_full), ("full_to_history", full_to_history),
                    ("header", header), ("checkin_iter", checkin_iter)):
        if t.dtype != torch.int64:
            raise TypeError(f"record_history_noalloc: {name} must be int64")
    if used_mask is not None:
        if used_mask.dtype not in (torch.bool, torch.uint8) or not used_mask.is_contiguous():
            raise TypeError("record_history_noalloc: used_mask must be contiguous bool")
        if used_mask.shape[0] < n:
            raise RuntimeError("record_history_noalloc: used_mask shorter than buffer_new")
    if sub_to_full.shape[0] < n or sub_to_history.shape[0] < n or score.shape[0] < n:
        raise RuntimeError("record_history_noalloc: per-row arguments shorter than buffer_new")
    if history_to_full.shape[0] < buffer_all.shape[0] or checkin_iter.shape[0] < buffer_all.shape[0]:
        raise RuntimeError("record_history_noalloc: slot arrays shorter than the table")
    with torch.cuda.device(dev):
        check(lib.hc_record_history_noalloc(
            ptr(buffer_new), hs, n, ptr(buffer_all), dtype_code(buffer_all), buffer_all.shape[0], hs,
            ptr(used_mask), ptr(sub_to_full), ptr(sub_to_history), ptr(history_to_full),
            ptr(full_to_history), ptr(header), ptr(score), ptr(thres), ptr(checkin_iter),
            int(glb_iter), ptr(n_admitted), stream_of(dev)), "hc_record_history_noalloc")
    _called(4)


CHECKIN_MARKER = 1 << 60   # a glb_iter no iteration takes


# ---------------------------------------------------------------------------
# receptive-field bookkeeping
# ---------------------------------------------------------------------------
count_history_reconstruct = _native.count_history_reconstruct
count_num = _native.count_num


def get_graph_structure_score(ptr_t, idx_t, num_node, num_seed, num_layer):
    """src/cpp/src/grad_check.cu:149-163 (level-synchronous, lowest-numbered parent wins)."""
    dev = require_cuda(ptr_t, idx_t)
    ptr_t, idx_t = i64c(ptr_t, "ptr"), i64c(idx_t, "idx")
    out = torch.empty(num_node, dtype=torch.int64, device=dev)
    sc = torch.empty(num_node, dtype=torch.int64, device=dev)
    with on_device(dev), _span("hc_structure_score", dev):
        check(lib.hc_structure_score(ptr(ptr_t), ptr(idx_t), ptr_t.shape[0] - 1, num_node,
                                     num_seed, num_layer, ptr(out), ptr(sc), stream_of(dev)),
              "hc_structure_score")
    _called()
    return out


# ---------------------------------------------------------------------------
# lookup and row assembly
# ---------------------------------------------------------------------------
map_lookup = _native.map_lookup
cache_lookup = _native.cache_lookup
gather_rows = _native.gather_rows
load_rows = _native.load_rows

# thread blocks of a staging call; non-zero overrides every caller's choice (a knob for measurements)
STAGE_BLOCKS = int(os.environ.get("HISCACHE_STAGE_BLOCKS", "0"))


def stage_host_rows(host_table, ids, sub2feat, consider, rows_out, mask_out, stats=None, max_blocks=None):
    """Copies host_table[ids[i]] into rows_out[i] and sets mask_out[i] for every i that is to be
    considered and is not in the feature cache (sub2feat[i] == -1); other rows of rows_out are
    unspecified.  The result feeds `load_rows(..., staged=(rows_out, mask_out))` of a later step."""
    _native.stage_host_rows(host_table, ids, sub2feat, consider, rows_out, mask_out, stats,
                            int(STAGE_BLOCKS or (max_blocks or 0)))


# ---------------------------------------------------------------------------
# sharded-table helpers
# ---------------------------------------------------------------------------
def mix64(x: int) -> int:
    return int(lib.hc_mix64(C.c_uint64(x & 0xFFFFFFFFFFFFFFFF)))


def bucket_by_owner(ids, world, keep=None):
    """Stable bucket sort by owner(id) = mix64(id) mod world: (counts, perm, bucketed)."""
    dev = require_cuda(ids, keep)
    ids = i64c(ids, "ids")
    n = ids.shape[0]
    counts = torch.empty(world, dtype=torch.int64, device=dev)
    perm = torch.empty(n, dtype=torch.int64, device=dev)
    bucketed = torch.empty(n, dtype=torch.int64, device=dev)
    sc = scratch(dev, lib.hc_bucket_scratch_bytes(n, world), "bucket")
    if keep is not None:
        keep = keep.contiguous()
    with on_device(dev), _span("hc_bucket_by_owner", dev):
        check(lib.hc_bucket_by_owner(ptr(ids), ptr(keep), n, world, ptr(counts), ptr(perm),
                                     ptr(bucketed), ptr(sc), stream_of(dev)), "hc_bucket_by_owner")
    _called(3)
    return counts, perm, bucketed


def bucket_pad(bucketed, counts, world, slots, overflow=None, out=None):
    """[world, slots] ids padded with -1 from bucket-ordered ids (no host sizes needed)."""
    dev = require_cuda(bucketed, counts)
    if out is None:
        out = torch.empty((world, slots), dtype=torch.int64, device=dev)
    with on_device(dev), _span("hc_bucket_pad", dev):
        check(lib.hc_bucket_pad(ptr(bucketed), ptr(counts), bucketed.shape[0], world, slots, ptr(out),
                                ptr(overflow), stream_of(dev)), "hc_bucket_pad")
    _called()
    return out


def unpad_hits(perm, counts, world, slots, flags_back=None, want_slots=False):
    """(hit_map, slot_of): row of the padded answer per original position, -1 for a miss."""
    dev = require_cuda(perm, counts)
    n = perm.shape[0]
    hit = torch.empty(n, dtype=torch.int64, device=dev) if flags_back is not None else None
    slot_of = torch.full((n,), -1, dtype=torch.int64, device=dev) if want_slots else None
    with on_device(dev), _span("hc_unpad_hits", dev):
        check(lib.hc_unpad_hits(ptr(perm), ptr(counts), n, world, slots, ptr(flags_back), ptr(hit),
                                ptr(slot_of), stream_of(dev)), "hc_unpad_hits")
    _called()
    return hit, slot_of


def last_occurrence(ids, claim):
    """uint8 mask: 1 where ids[k] >= 0 does not appear again later.  claim: int32 [N] of -1."""
    dev = require_cuda(ids, claim)
    ids = i64c(ids, "ids")
    if claim.dtype != torch.int32:
        raise TypeError("claim must be int32")
    win = torch.empty(ids.shape[0], dtype=torch.uint8, device=dev)
    with on_device(dev), _span("hc_last_occurrence", dev):
        check(lib.hc_last_occurrence(ptr(ids), ids.shape[0], ptr(claim), claim.shape[0], ptr(win),
                                     stream_of(dev)), "hc_last_occurrence")
    _called(3)
    return win


def unpermute_rows(src, perm, flags, dst, hit_out=None):
    """dst[perm[k]] = src[k] where flags[k]; hit_out[perm[k]] = k or -1."""
    dev = require_cuda(perm, src, dst, hit_out)
    n = perm.shape[0]
    F = 0 if src is None else src.shape[1]
    if flags is not None:
        flags = flags.contiguous()
    with on_device(dev), _span("hc_unpermute_rows", dev):
        check(lib.hc_unpermute_rows(ptr(src), HC_F32 if src is None else dtype_code(src),
                                    0 if src is None else (src.stride(0) if n > 1 else F), F,
                                    ptr(i64c(perm)), ptr(flags), n, ptr(dst),
                                    0 if dst is None else (dst.stride(0) if dst.shape[0] > 1 else F),
                                    ptr(hit_out), stream_of(dev)), "hc_unpermute_rows")
    _called()


def owner_lookup(map_t, ids, table, rows_out=None):
    """Owner-side lookup of the exchange: (flags, rows_out)."""
    dev = require_cuda(map_t, ids, table)
    ids = i64c(ids, "ids")
    n = ids.shape[0]
    flags = torch.empty(n, dtype=torch.uint8, device=dev)
    F = table.shape[1]
    if rows_out is None:
        rows_out = torch.empty((n, F), dtype=table.dtype, device=dev)
    with on_device(dev), _span("hc_owner_lookup", dev):
        check(lib.hc_owner_lookup(ptr(map_t), map_t.shape[0], ptr(ids), n, ptr(table),
                                  dtype_code(table), table.shape[0],
                                  table.stride(0) if table.shape[0] > 1 else F, F, ptr(rows_out),
                                  rows_out.stride(0) if n > 1 else F, ptr(flags), stream_of(dev)),
              "hc_owner_lookup")
    _called()
    return flags, rows_out


# ---------------------------------------------------------------------------
# history exchange over peer memory
# ---------------------------------------------------------------------------
HC_MAX_PEERS = 32


class PeerRegion:
    """One device allocation made by the library (hc_peer_alloc) that other processes of the
    box can map.  `view(offset, shape, dtype)` gives torch tensors over parts of it."""

    def __init__(self, nbytes, device):
        self.device = torch.device(device)
        self.nbytes = int(nbytes)
        out = C.c_void_p()
        with torch.cuda.device(self.device):
            check(lib.hc_peer_alloc(self.nbytes, C.byref(out)), "hc_peer_alloc")
        self.ptr = int(out.value)
        self.__cuda_array_interface__ = {"shape": (self.nbytes,), "typestr": "|u1",
                                         "data": (self.ptr, False), "version": 2}
        with torch.cuda.device(self.device):
            self.bytes = torch.as_tensor(self, device=self.device)
        if self.bytes.data_ptr() != self.ptr:
            raise RuntimeError("PeerRegion: torch copied the region instead of viewing it")

    def view(self, offset, shape, dtype):
        n = 1
        for d in shape:
            n *= int(d)
        nb = n * torch.empty((), dtype=dtype).element_size()
        if offset % 16 or offset + nb > self.nbytes:
            raise ValueError("PeerRegion.view: bad offset or size")
        return self.bytes[offset:offset + nb].view(dtype).view(*shape)

    def export(self) -> bytes:
        buf = C.create_string_buffer(64)
        with torch.cuda.device(self.device):
            check(lib.hc_peer_export(self.ptr, buf), "hc_peer_export")
        return buf.raw

    def free(self):
        if self.ptr:
            self.bytes = None
            with torch.cuda.device(self.device):
                check(lib.hc_peer_free(self.ptr), "hc_peer_free")
            self.ptr = 0


def peer_open(handle: bytes, device) -> int:
    """Maps another process's exported region into this one; returns its device address."""
    if len(handle) != 64:
        raise ValueError("peer_open: a handle is 64 bytes")
    out = C.c_void_p()
    with torch.cuda.device(device):
        check(lib.hc_peer_open(C.create_string_buffer(handle, 64), C.byref(out)), "hc_peer_open")
    return int(out.value)


def peer_close(address: int, device):
    with torch.cuda.device(device):
        check(lib.hc_peer_close(address), "hc_peer_close")


def peer_ptrs(addresses):
    """Host pointer table (one device address per rank) in the form the peer calls take."""
    if not 1 <= len(addresses) <= HC_MAX_PEERS:
        raise ValueError(f"between 1 and {HC_MAX_PEERS} ranks")
    return (C.c_void_p * len(addresses))(*[int(a) for a in addresses])


def peer_lookup(maps, tables, world, map_len, table_rows, feat, dtype, ids, rows_out=None):
    """One-kernel lookup in the node-partitioned history: (hit_map [n], rows [n, feat]).
    maps / tables: peer_ptrs() of every rank's id->slot map and row table."""
    dev = require_cuda(ids)
    ids = i64c(ids, "ids")
    n = ids.shape[0]
    if rows_out is None:
        rows_out = torch.empty((n, feat), dtype=dtype, device=dev)
    hit = torch.empty(n, dtype=torch.int64, device=dev)
    with on_device(dev), _span("hc_peer_lookup", dev):
        check(lib.hc_peer_lookup(maps, tables, world, map_len, dtype_code(rows_out), table_rows, feat,
                                 feat, ptr(ids), n, ptr(rows_out), rows_out.stride(0) if n > 1 else feat,
                                 ptr(hit), stream_of(dev)), "hc_peer_lookup")
    _called()
    return hit, rows_out


def peer_publish(ids, rows, mask, pub_ids, pub_rows, pub_n, score=None, thres=None, present=None):
    """Writes this rank's admission candidates into its published area: rows with mask set
    (None = all), score < thres (when given) and present == -1 (when given)."""
    dev = require_cuda(ids, rows, mask, pub_ids, pub_rows, pub_n, score, thres, present)
    if score is not None:
        if thres is None or score.dtype != torch.float32 or thres.dtype != torch.float32:
            raise TypeError("peer_publish: score and thres must be float32 tensors")
        score = score.contiguous()
        if score.shape[0] != ids.shape[0]:
            raise ValueError("peer_publish: one score per id")
    present = i64c(present, "present")
    if present is not None and present.shape[0] != ids.shape[0]:
        raise ValueError("peer_publish: one present entry per id")
    ids = i64c(ids, "ids")
    n = ids.shape[0]
    if rows.dtype != torch.float32:
        raise TypeError("peer_publish: rows must be float32")
    rows = rows2d(rows)
    if mask is not None:
        mask = mask.contiguous()
        if mask.dtype == torch.bool:
            mask = mask.view(torch.uint8)
    F = pub_rows.shape[1]
    if n and rows.shape[1] != F:
        raise ValueError("peer_publish: row width differs from the published area")
    with on_device(dev), _span("hc_peer_publish", dev):
        check(lib.hc_peer_publish(ptr(ids), ptr(mask), ptr(score), ptr(thres), ptr(present), n, ptr(rows),
                                  rows.stride(0) if n > 1 else F, F,
                                  ptr(pub_ids), ptr(pub_rows), ptr(pub_n), pub_ids.shape[0],
                                  stream_of(dev)), "hc_peer_publish")
    _called()


def peer_pull(pub_ids, pub_rows, pub_n, world, me, max_ids, feat, got_ids, got_rows, overflow=None):
    """Collects, in (rank, row) order, the published candidates this rank owns into
    got_ids [cap] (tail -1) and got_rows [cap, feat] fp32."""
    dev = require_cuda(got_ids, got_rows, overflow)
    cap = got_ids.shape[0]
    sc = scratch(dev, int(lib.hc_peer_pull_scratch_bytes(world, max_ids)), "peer_pull")
    with on_device(dev), _span("hc_peer_pull", dev):
        check(lib.hc_peer_pull(pub_ids, pub_rows, pub_n, world, me, max_ids, feat, ptr(got_ids),
                               ptr(got_rows), cap, ptr(overflow), ptr(sc), stream_of(dev)), "hc_peer_pull")
    _called(3)
    return got_ids, got_rows


def make_shard(full_to_slot, slot_to_full, checkin, table, header, iter_dev, claim, staleness,
               n_admitted=None):
    """struct hc_shard over one rank's tables (keep the tensors alive while it is used)."""
    require_cuda(full_to_slot, slot_to_full, checkin, table, header, iter_dev, claim, n_admitted)
    if claim.dtype != torch.int32:
        raise TypeError("claim must be int32")
    for t, name in ((full_to_slot, "full_to_slot"), (slot_to_full, "slot_to_full"), (checkin, "checkin"),
                    (header, "header"), (iter_dev, "iter_dev")):
        if t.dtype != torch.int64 or not t.is_contiguous():
            raise TypeError(f"{name} must be contiguous int64")
    if not table.is_contiguous():
        raise ValueError("table must be contiguous")
    sh = _capi.Shard()
    sh.struct_size = C.sizeof(_capi.Shard)
    sh.full_to_slot, sh.map_len = ptr(full_to_slot), full_to_slot.shape[0]
    sh.slot_to_full, sh.checkin, sh.capacity = ptr(slot_to_full), ptr(checkin), table.shape[0]
    sh.table, sh.dtype, sh.feat = ptr(table), dtype_code(table), table.shape[1]
    sh.header, sh.iter_dev, sh.claim = ptr(header), ptr(iter_dev), ptr(claim)
    sh.staleness, sh.n_admitted = int(staleness), ptr(n_admitted)
    return sh


def peer_admit(shard, pub_ids, pub_rows, pub_n, world, me, max_ids, got_ids, got_rows, overflow=None,
               evict=True, advance_iter=False):
    """Owner-side admission of one step in one call (evict, pull, last copy wins, skip ids
    already held, ring admission, stamp, optional iteration advance)."""
    dev = require_cuda(got_ids, got_rows, overflow)
    cap = got_ids.shape[0]
    sc = scratch(dev, int(lib.hc_peer_admit_scratch_bytes(world, max_ids, cap)), "peer_admit")
    with on_device(dev), _span("hc_peer_admit", dev):
        check(lib.hc_peer_admit(C.byref(shard), pub_ids, pub_rows, pub_n, world, me, max_ids, ptr(got_ids),
                                ptr(got_rows), cap, ptr(overflow), 1 if evict else 0,
                                1 if advance_iter else 0, ptr(sc), stream_of(dev)), "hc_peer_admit")
    _called(14)


# ---------------------------------------------------------------------------
# neighbour sampling (stand-in for the external loader)
# ---------------------------------------------------------------------------
ABSENT = -(1 << 31)  # local_map value of a node outside the batch

sample_hop = _native.sample_hop
relabel_seed = _native.relabel_seed
relabel_reset = _native.relabel_reset
relabel = _native.relabel


def sample_fixed(gptr, gidx, seeds, local_map, seed, batch_no, fanouts, caps, edge_cap, out=None, labels=None):
    """A whole batch in the fixed shape (caps, edge_cap) without any device->host read
    (hc_sample_fixed).  `batch_no`: device int64[1], advanced by the call.  Returns the dict of
    output tensors (ptr, idx, sub_to_full, mask, counters); `out` reuses a previous one.  With `labels`
    (int64 per node) out["y"] is filled too: the seeds' labels, -100 in padding rows."""
    L = len(fanouts)
    if len(caps) != L + 1 or L < 1 or L > 8:
        raise ValueError("sample_fixed: one cap per layer (hops + 1), 1..8 hops")
    if local_map.dtype != torch.int32 or batch_no.dtype != torch.int64:
        raise TypeError("sample_fixed: local_map int32, batch_no int64")
    if seeds.shape[0] > caps[0]:
        raise RuntimeError("sample_fixed: more seeds than caps[0]")
    if out is None:
        dev = require_cuda(gptr)
        out = {"ptr": torch.empty(caps[L - 1] + 1, dtype=torch.int64, device=dev),
               "idx": torch.empty(max(int(edge_cap), 1), dtype=torch.int64, device=dev),
               "sub_to_full": torch.empty(caps[L], dtype=torch.int64, device=dev),
               "mask": torch.empty(caps[L], dtype=torch.bool, device=dev),
               "counters": torch.zeros(4, dtype=torch.int64, device=dev)}
    if labels is not None and "y" not in out:
        out["y"] = torch.empty(caps[0], dtype=torch.int64, device=gptr.device)
    _native.sample_batch(gptr, gidx, seeds, local_map, int(seed) & 0xFFFFFFFFFFFFFFFF, batch_no, fanouts, caps,
                         int(edge_cap), out["ptr"], out["idx"], out["sub_to_full"], out["mask"], out["counters"],
                         labels, None if labels is None else out["y"])
    return out


# ---------------------------------------------------------------------------
# heterogeneous layers
# ---------------------------------------------------------------------------
edge_types = _native.edge_types
rgcn_group = _native.rgcn_group
RGCN_ROWS_MAX_REL = 8


def rgcn_layer(x, ptr, idx, edge_type, num_node, weight, *, used_src=None, history_map=None, history_buffer=None,
               indexed=False):
    """One RGCN layer: out[d] = (1/deg(d)) * sum_e x[src_e] @ weight[rel_e], history rows over it.
    Returns (out, edges per relation [num_rel + 1] with value 0 never counted, pruned slots last).
    weight [num_rel, feat, hidden] fp32, at most RGCN_ROWS_MAX_REL relations."""
    return _native.rgcn_layer(x, ptr, idx, edge_type, int(num_node), used_src, history_map, history_buffer, indexed,
                              weight, DETERMINISTIC_BWD, GATHER_MIN_BYTES, GATHER_MIN_FEAT)


# ---------------------------------------------------------------------------
# dense part of a SAGE layer, loss, optimiser
# ---------------------------------------------------------------------------
def nll_loss(logp, y, ignore_index=-100):
    """torch.nn.functional.nll_loss (mean over the labelled rows), one kernel per direction."""
    if logp.dim() == 2 and y.dim() == 1 and logp.dtype == torch.float32 and y.dtype == torch.int64:
        return _native.nll_loss(logp, y, ignore_index)
    return torch.nn.functional.nll_loss(logp, y, ignore_index=ignore_index)


sage_linear = _native.sage_linear       # (his, x, num_node, w_l, bias, w_r, slabs)
adam_step = _native.adam_step           # (params, grads, exp_avgs, exp_avg_sqs, steps, lr, beta1, beta2, eps) -> whether done
adam_fits = _native.adam_fits           # (params, grads, exp_avgs, exp_avg_sqs, steps) -> bool

# ---------------------------------------------------------------------------
# peer copies (kept for API compatibility; the multi-GPU path uses NCCL)
# ---------------------------------------------------------------------------
def p2psend(tsrc, tdst, num_element, target_device):
    """src/cpp/src/comm.cu:3-11: copies the first num_element elements of tsrc into tdst,
    which lives on target_device.  Unlike the reference the current device is left
    unchanged and the element size follows the dtype."""
    tdst.view(-1)[:num_element].copy_(tsrc.reshape(-1)[:num_element], non_blocking=True)


def p2psend_gentensor(tsrc, num_element, target_device):
    """src/cpp/src/comm.cu:13-20: allocates the destination on target_device first."""
    tdst = torch.empty_like(tsrc, device=torch.device("cuda", int(target_device)))
    p2psend(tsrc, tdst, num_element, target_device)
    return tdst
