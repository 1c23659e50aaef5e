"""Layer-level operators against plain torch: the RGCN layer, the dense part of a SAGE layer with the
aggregation's rooted backward, and the Adam step."""
import numpy as np
import pytest
import torch

from _gen import layered_batch

pytestmark = pytest.mark.gpu


def cu(a):
    return None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()


def block(seed, seeds, fanout, total):
    b = layered_batch(np.random.default_rng(seed), seeds, fanout, total_nodes=total)
    return b["ptr"], b["idx"], [int(v) for v in b["num_node_in_layer"]]


@pytest.mark.parametrize("seeds,rel,feat,hidden,dt", [
    (1, 1, 4, 3, torch.float32), (17, 5, 36, 20, torch.float32), (60, 8, 33, 16, torch.float32),
    (300, 3, 128, 64, torch.float16)])
@pytest.mark.parametrize("used,hist", [(False, None), (True, "rows"), (True, "indexed")])
def test_rgcn_layer(backend, oracle, seeds, rel, feat, hidden, dt, used, hist):
    ptr, idx, nn = block(3 + seeds, seeds, [25, 15], 9000)
    num_node, n_all = nn[1], nn[-1]
    rng = np.random.default_rng(5)
    et = rng.integers(0, rel, size=len(idx)).astype(np.int64)
    us = (rng.random(n_all) < 0.7) if used else None
    hm = np.where(rng.random(num_node) < 0.3, rng.integers(0, 50, num_node), -1).astype(np.int64) if hist else None
    hb = None
    if hist:
        hb = torch.randn(50 if hist == "indexed" else num_node, hidden, device="cuda")
        if seeds == 300:
            hb = hb.half()
    x = (torch.randn(n_all, feat, device="cuda") * 0.5).to(dt).requires_grad_()
    w = (torch.randn(rel, feat, hidden, device="cuda") * 0.2).requires_grad_()
    out, count = backend.rgcn_layer(x, cu(ptr), cu(idx), cu(et), num_node, w, used_src=cu(us), history_map=cu(hm),
                                    history_buffer=hb, indexed=hist == "indexed")
    g = torch.randn_like(out)
    out.backward(g)

    src, dst, rel_w, perm, _ = oracle.rgcn_sorted_edges(ptr, idx, et, num_node, rel, us, hm)
    keep = int((rel_w < rel).sum())
    src, dst, r = cu(src[:keep]), cu(dst[:keep]), cu(rel_w[perm[:keep]])
    xd, wd = x.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    deg = cu(np.diff(ptr)[:num_node]).double()
    want = torch.zeros(num_node, hidden, dtype=torch.float64, device="cuda")
    want = want.index_add(0, dst, torch.einsum("ef,efh->eh", xd[src], wd[r]) / deg[dst][:, None]) \
        if keep <= 20000 else want + sum(
            torch.zeros(num_node, feat, dtype=torch.float64, device="cuda").index_add(
                0, dst[r == k], xd[src[r == k]] / deg[dst[r == k]][:, None]) @ wd[k] for k in range(rel))
    if hist:
        hmt = cu(hm)
        rows = hb[hmt.clamp(min=0)] if hist == "indexed" else hb
        want = torch.where((hmt != -1)[:, None], rows.double(), want)
    want.backward(g.double())
    for a, b in ((out, want), (x.grad, xd.grad), (w.grad, wd.grad)):
        tol = 2e-3 if a.dtype == torch.float16 else 2e-5
        assert (a.double() - b).abs().max() <= tol * (1 + b.abs().max())
    c = np.bincount(rel_w[rel_w < rel], minlength=rel)
    c[0] = 0
    assert np.array_equal(count.cpu().numpy()[:rel], c)
    assert int(count[rel]) == len(idx) - keep
