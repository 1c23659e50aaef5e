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


@pytest.mark.parametrize("feat,hidden,seeds,bias", [(8, 12, 3, True), (100, 256, 40, True), (33, 7, 9, False),
                                                    (256, 47, 200, True)])
@pytest.mark.parametrize("mode", ["scatter", "source", "deterministic"])
@pytest.mark.parametrize("dt", [torch.float32, torch.float16])
def test_sage_linear_takes_both_gradients_along(backend, monkeypatch, feat, hidden, seeds, bias, mode, dt):
    monkeypatch.setattr(backend, "DETERMINISTIC_BWD", mode == "deterministic")
    monkeypatch.setattr(backend, "GATHER_MIN_BYTES", 0 if mode == "source" else 1 << 60)
    monkeypatch.setattr(backend, "GATHER_MIN_FEAT", 0)
    ptr, idx, nn = block(seeds, seeds, [10, 5], 5000)
    n, n_all = nn[1], nn[-1]
    x = (torch.randn(n_all, feat, device="cuda")).to(dt).requires_grad_()
    wl = (torch.randn(hidden, feat, device="cuda") * 0.1).requires_grad_()
    wr = (torch.randn(hidden, feat, device="cuda") * 0.1).requires_grad_()
    b = torch.randn(hidden, device="cuda").requires_grad_() if bias else None
    his = backend.aggr_forward(x, cu(ptr), cu(idx), n)
    his.retain_grad()
    out = backend.sage_linear(his, x, n, wl, b, wr, 8)
    g = torch.randn_like(out)
    params = [p for p in (x, wl, wr, b) if p is not None]
    out.backward(g, retain_graph=True)
    first = [p.grad.clone() for p in params]
    for p in params:
        p.grad = None
    out.backward(g)                       # a second pass over the same graph gives the same
    d = [p.detach().double().requires_grad_() for p in params]
    deg = np.diff(ptr)[:n]
    e = int(ptr[n])
    dst = cu(np.repeat(np.arange(n), deg))
    hd = torch.zeros(n, feat, dtype=torch.float64, device="cuda").index_add(0, dst, d[0][cu(idx[:e])])
    hd = hd / cu(np.maximum(deg, 1)).double()[:, None]
    hd.retain_grad()
    want = hd @ d[1].t() + d[0][:n] @ d[2].t() + (d[3] if bias else 0)
    want.backward(g.double())
    assert (out.double() - want).abs().max() <= 2e-5 * (1 + want.abs().max())
    assert (his.grad.double() / 2 - hd.grad).abs().max() <= 2e-5 * (1 + hd.grad.abs().max())
    for got, again, w in zip(first, params, d):
        tol = 2e-3 if got.dtype == torch.float16 else 3e-5
        assert (got.double() - w.grad).abs().max() <= tol * (1 + w.grad.abs().max())
        assert (again.grad.double() - w.grad).abs().max() <= tol * (1 + w.grad.abs().max())


def test_sage_linear_with_an_unrelated_aggregate(backend):
    x = torch.randn(50, 12, device="cuda", requires_grad=True)
    his = torch.randn(20, 12, device="cuda", requires_grad=True)
    wl, wr = (torch.randn(5, 12, device="cuda", requires_grad=True) for _ in range(2))
    out = backend.sage_linear(his, x, 20, wl, None, wr, 8)
    g = torch.randn_like(out)
    out.backward(g)
    assert torch.allclose(out, his @ wl.t() + x[:20] @ wr.t(), atol=1e-4)
    assert torch.allclose(his.grad, g @ wl, atol=1e-4)
    assert torch.allclose(x.grad[:20], g @ wr, atol=1e-4) and not x.grad[20:].any()


@pytest.mark.parametrize("sizes", [[1], [3, 1024, 1025, 5000], [64] * 49 + [70000]])
def test_adam_step_matches_torch(backend, sizes):
    from hiscache.optim import Adam
    init = [torch.randn(n, device="cuda") for n in sizes]
    a, b = ([t.clone().requires_grad_() for t in init] for _ in range(2))
    ours = Adam(a, lr=3e-3, betas=(0.8, 0.95), fused=True, capturable=True)
    theirs = torch.optim.Adam(b, lr=3e-3, betas=(0.8, 0.95), fused=True, capturable=True)
    for step in range(4):
        for k, (p, q) in enumerate(zip(a, b)):
            p.grad = torch.randn_like(p) if (k + step) % 3 or len(sizes) == 1 else None
            q.grad = None if p.grad is None else p.grad.clone()
        version = a[0]._version
        ours.step()
        theirs.step()
        assert a[0].grad is None or a[0]._version > version
    for p, q in zip(a, b):
        assert torch.allclose(p, q, rtol=1e-6, atol=1e-8)
    so, st = ours.state_dict(), theirs.state_dict()
    assert so["state"].keys() == st["state"].keys()
    for k in so["state"]:
        for name in ("step", "exp_avg", "exp_avg_sq"):
            assert torch.allclose(so["state"][k][name], st["state"][k][name], rtol=1e-5, atol=1e-7)
    ours.load_state_dict(st)
    assert isinstance(ours, torch.optim.Adam)


@pytest.mark.parametrize("n,hidden,feat", [
    (1, 3, 5), (255, 47, 100), (512, 64, 33), (2051, 256, 128), (5000, 1100, 8), (9473, 47, 50)])
def test_dense_part_of_a_layer(backend, n, hidden, feat):
    """Row counts that are no multiple of the slabs, outputs wider than a block, one slab."""
    x = torch.randn(n + 3, feat, device="cuda", requires_grad=True)
    his = torch.randn(n, feat, device="cuda", requires_grad=True)
    wl, wr = (torch.randn(hidden, feat, device="cuda", requires_grad=True) for _ in range(2))
    b = torch.randn(hidden, device="cuda", requires_grad=True)
    g = torch.randn(n, hidden, device="cuda")
    d = [t.detach().double() for t in (his, x, wl, wr, b, g)]
    zero = torch.zeros(3, feat, dtype=torch.float64, device="cuda")
    want_grads = (d[5] @ d[2], torch.cat([d[5] @ d[3], zero]), d[5].t() @ d[0], d[5].t() @ d[1][:n], d[5].sum(0))
    for bias in (b, None):
        for slabs in (1, 8):
            out = backend.sage_linear(his, x, n, wl, bias, wr, slabs)
            want = d[0] @ d[2].t() + d[1][:n] @ d[3].t() + (d[4] if bias is not None else 0)
            assert (out - want).abs().max() <= 1e-5 * (1 + want.abs().max())
            over = (his, x, wl, wr) + (() if bias is None else (b,))
            for a, w in zip(torch.autograd.grad(out, over, g), want_grads):
                assert (a - w).abs().max() <= 1e-5 * (1 + w.abs().max())
    only = torch.autograd.grad(backend.sage_linear(his.detach(), x.detach(), n, wl.detach(), b, wr, 8), (b, wr), g)
    assert (only[0] - want_grads[4]).abs().max() <= 1e-5 * (1 + want_grads[4].abs().max())
    assert (only[1] - want_grads[3]).abs().max() <= 1e-5 * (1 + want_grads[3].abs().max())


@pytest.mark.parametrize("n,classes", [(1, 2), (1000, 172), (1025, 47), (9000, 153)])
@pytest.mark.parametrize("ignored", [0.0, 0.3, 1.0])
def test_nll_loss(backend, n, classes, ignored):
    logp = torch.randn(n, classes + 1, device="cuda").log_softmax(-1)[:, :classes].requires_grad_()
    y = torch.randint(0, classes, (n,), device="cuda")
    y[torch.rand(n, device="cuda") < ignored] = -100
    loss = backend.nll_loss(logp, y)
    want = torch.nn.functional.nll_loss(logp.double(), y)
    if bool((y == -100).all()):
        assert torch.isnan(loss) and torch.isnan(want)
        return
    assert loss.shape == want.shape and abs(float(loss) - float(want)) <= 1e-6 * abs(float(want))
    got, = torch.autograd.grad(loss * 3, logp)
    ref, = torch.autograd.grad(want * 3, logp)
    assert torch.allclose(got, ref.float(), rtol=1e-6, atol=0)
