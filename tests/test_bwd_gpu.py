"""GPU parity tests of the backward kernels (attention and indexer), called through the C ABI,
against the oracle's restatement of the reference's backward kernels and against gradients the
reference itself produced (fixtures)."""
import os

import numpy as np
import pytest
import torch

from oracle import dsa as O

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.fixture(scope="module")
def swv():
    import sparse_wsi_vit_b200 as m
    return m


def _close(a, b, rel=2e-4):
    ref = float(b.abs().max())
    return float((a.cpu().float() - b).abs().max()) <= rel * max(1.0, ref)


@pytest.mark.parametrize("case", ["bwd_rand", "bwd_batch2", "bwd_short"])
def test_backward_kernels_match_reference_gradients(swv, golden_dir, case):
    g = np.load(os.path.join(golden_dir, "dsa_bwd_reference.npz"))
    B, T, H, D, IH, ID, K = [int(x) for x in g[f"{case}.dims"]]
    t = lambda n: torch.from_numpy(g[f"{case}.{n}"])
    d = lambda n: t(n).to(DEV)
    rw = d("scores") * d("valid")
    dq, dk, dv, drw = swv.ops.dsa_attention_bwd(d("d_out"), d("q"), d("k"), d("v"), d("o"), d("idx"), d("valid"), rw)
    swv.check_status(DEV)
    for mine, name in ((dq, "dq"), (dk, "dk"), (dv, "dv"), (drw, "drw")):
        assert _close(mine, t(name)), (case, name)
    dqi, dki, dw = swv.ops.dsa_indexer_bwd(d("drw") * d("valid"), d("qi"), d("ki"), d("w"), d("idx"), d("valid"))
    swv.check_status(DEV)
    assert _close(dqi, t("dqi")) and _close(dki, t("dki")) and _close(dw, t("dw"), rel=1e-3), case


@pytest.mark.parametrize("T,Tk,H,D,K,dtype", [(200, 200, 2, 64, 32, torch.float32), (77, 300, 1, 32, 8, torch.float32),
                                              (130, 130, 2, 128, 64, torch.bfloat16), (50, 50, 3, 64, 5000, torch.float32),
                                              (64, 64, 1, 160, 16, torch.bfloat16)])
def test_attention_backward_vs_oracle(swv, T, Tk, H, D, K, dtype):
    """Unsorted lists with a repeated key and an invalid slot; cross lengths (queries are a slice of
    the keys); top_k beyond the logit cache (recompute path); head dims 32..160; bf16 inputs."""
    g = torch.Generator().manual_seed(T + K)
    q = (torch.randn(1, H, T, D, generator=g) / D ** 0.5).to(dtype)
    k = torch.randn(1, H, Tk, D, generator=g).to(dtype)
    v = torch.randn(1, H, Tk, D, generator=g).to(dtype)
    keff = min(K, Tk)
    idx = torch.zeros(1, T, K, dtype=torch.int32)
    valid = torch.zeros(1, T, K)
    for r in range(T):
        idx[0, r, :keff] = torch.randperm(Tk, generator=g)[:keff].to(torch.int32)
    valid[..., :keff] = 1.0
    idx[:, :, 1] = idx[:, :, 0]
    valid[:, :, 2] = 0.0
    rw = torch.rand(1, T, K, generator=g) * valid
    d_out = torch.randn(1, H, T, D, generator=g)
    o = O.dsa_attention(q[0].float(), k[0].float(), v[0].float(), idx[0], valid[0], rw[0])[None]
    dq, dk, dv, drw = swv.ops.dsa_attention_bwd(d_out.to(DEV), q.to(DEV), k.to(DEV), v.to(DEV), o.to(DEV), idx.to(DEV),
                                                valid.to(DEV), rw.to(DEV))
    swv.check_status(DEV)
    rq, rk, rv, rrw = O.dsa_attention_bwd(d_out[0], q[0].float(), k[0].float(), v[0].float(), o[0], idx[0], valid[0],
                                          rw[0])
    assert _close(dq[0], rq) and _close(dk[0], rk) and _close(dv[0], rv) and _close(drw[0], rrw)


@pytest.mark.parametrize("B,T,Tk,IH,ID,K,dtype", [(1, 150, 150, 4, 64, 16, torch.float32), (2, 60, 200, 2, 16, 8, torch.bfloat16),
                                                  (1, 40, 40, 4, 32, 64, torch.float32), (1, 33, 90, 8, 64, 12, torch.bfloat16)])
def test_indexer_backward_vs_oracle(swv, B, T, Tk, IH, ID, K, dtype):
    g = torch.Generator().manual_seed(B * 100 + T)
    qi = (torch.randn(B, T, IH, ID, generator=g) / ID ** 0.5).to(dtype)
    ki = (torch.randn(B, Tk, IH, ID, generator=g) / ID ** 0.5).to(dtype)
    w = torch.randn(IH, generator=g)
    keff = min(K, Tk)
    idx = torch.zeros(B, T, K, dtype=torch.int32)
    valid = torch.zeros(B, T, K)
    for b in range(B):
        for r in range(T):
            idx[b, r, :keff] = torch.randperm(Tk, generator=g)[:keff].to(torch.int32)
    valid[..., :keff] = 1.0
    ds = torch.randn(B, T, K, generator=g)
    dq, dk, dw = swv.ops.dsa_indexer_bwd(ds.to(DEV), qi.to(DEV), ki.to(DEV), w.to(DEV), idx.to(DEV), valid.to(DEV))
    swv.check_status(DEV)
    dw_ref = torch.zeros(IH)
    for b in range(B):
        rq, rk, rw_ = O.indexer_bwd(ds[b], qi[b].float(), ki[b].float(), w, idx[b], valid[b])
        assert _close(dq[b], rq) and _close(dk[b], rk)
        dw_ref += rw_
    assert _close(dw, dw_ref, rel=1e-3)


def test_autograd_functions_and_module_train_step(swv):
    """The two reference-shaped autograd Functions chained the way the reference module chains them,
    and the module's own differentiable path (fused forward): gradients reach q/k/v, the indexer
    projections and the head weights, and agree with the oracle's backward on the same lists."""
    B, T, H, D, IH, ID, K = 1, 300, 2, 64, 4, 32, 48
    g = torch.Generator().manual_seed(9)
    mk = lambda *s, sc=1.0: (torch.randn(*s, generator=g) * sc).to(DEV).requires_grad_()
    q, k, v = mk(B, H, T, D, sc=0.125), mk(B, H, T, D), mk(B, H, T, D)
    qi, ki = mk(B, T, IH, ID, sc=0.18), mk(B, T, IH, ID, sc=0.18)
    w = mk(IH)
    d_out = torch.randn(B, H, T, D, generator=g).to(DEV)
    idx, valid, scores = swv.LightningIndexerFunction.apply(qi, ki, w, B, T, IH, ID, K, 16, 16, 16, IH)
    rw = scores * valid
    o = torch.zeros(B, H, T, D, device=DEV)
    out = swv.DSAAttentionFunction.apply(q, k, v, idx.detach(), valid.detach(), rw, o, B, H, T, D, K, 16, 16, H, 16)
    (out * d_out).sum().backward()
    swv.check_status(DEV)
    c = lambda x: x.detach().cpu()
    rq, rk, rv, rrw = O.dsa_attention_bwd(c(d_out)[0], c(q)[0], c(k)[0], c(v)[0], c(out)[0], c(idx)[0], c(valid)[0],
                                          c(rw)[0])
    assert _close(q.grad[0], rq) and _close(k.grad[0], rk) and _close(v.grad[0], rv)
    rqi, rki, rdw = O.indexer_bwd(rrw * c(valid)[0], c(qi)[0], c(ki)[0], c(w), c(idx)[0], c(valid)[0])
    assert _close(qi.grad[0], rqi) and _close(ki.grad[0], rki) and _close(w.grad, rdw, rel=1e-3)

    # the module: bf16 fused forward, one differentiable op; every parameter gets a finite gradient
    torch.manual_seed(0)
    m = swv.DeepSeekSparseAttention(d_model=128, attention_heads=2, indexer_heads=4, indexer_dim=32, top_k=64).to(DEV)
    x = torch.randn(1, 400, 128, generator=torch.Generator().manual_seed(1)).to(DEV).requires_grad_()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = m(x)
    y.float().square().mean().backward()
    swv.check_status(DEV)
    assert torch.isfinite(x.grad).all() and float(x.grad.abs().max()) > 0
    for n, p_ in m.named_parameters():
        assert p_.grad is not None and torch.isfinite(p_.grad).all(), n
    assert float(m.indexer_head_weights.grad.abs().max()) > 0
    # against the fp32 gather-path Functions on the same weights and lists
    m32 = m.float()
    x2 = x.detach().clone().requires_grad_()
    y2 = m32(x2)
    assert (y2 - y.float()).abs().max() < 5e-2


def test_encoder_train_steps_reduce_the_loss(swv):
    """Three optimisation steps of a small DSA encoder through ``training.train_step`` (bf16 autocast,
    the backward kernels under autograd) on a fixed ragged batch: finite gradients everywhere and a
    falling loss."""
    from sparse_wsi_vit_b200.training import train_step
    torch.manual_seed(0)
    net = swv.DSAViTSlideEncoder(in_features=64, out_features=2, embed_dim=128, num_heads=2, num_layers=2, num_cls=2,
                                 indexer_heads=4, indexer_dim=32, top_k=64, rope_coord_high=224.0 * 16).to(DEV).train()
    g = torch.Generator().manual_seed(1)
    batch = {"input": [torch.randn(n, 64, generator=g).to(DEV) for n in (300, 450)],
             "coords": [(torch.randint(0, 16, (n, 2), generator=g) * 224).float().to(DEV) for n in (300, 450)],
             "label": torch.tensor([0, 1], device=DEV)}
    opt = torch.optim.AdamW(net.parameters(), lr=2e-3)
    losses = [train_step(net, opt, batch) for _ in range(4)]
    swv.check_status(DEV)
    assert all(np.isfinite(l) for l in losses), losses
    assert losses[-1] < losses[0], losses
    for n, p_ in net.named_parameters():
        assert p_.grad is not None and torch.isfinite(p_.grad).all(), n


@pytest.mark.parametrize("B,T,H,IH,ID,K,o_dtype,exact", [
    (1, 64, 1, 4, 32, 16, torch.bfloat16, True),      # less than one tile
    (1, 128, 2, 4, 64, 128, torch.float32, True),     # every key selected, exactly one tile
    (2, 300, 3, 4, 32, 40, torch.float32, True),      # ragged tiles, batch, fp32 output with bf16-exact gradients
    (1, 517, 2, 4, 64, 96, torch.float32, False),     # gradients with more bits than bf16: the list kernel takes over
    (1, 260, 1, 2, 32, 300, torch.bfloat16, True),    # more slots than keys, one 64-channel projection block
    (1, 391, 2, 3, 64, 33, torch.bfloat16, True),     # 192 projection channels: indexer gradients on the list kernel
    (2, 1100, 1, 4, 32, 48, torch.bfloat16, True),    # few tiles: the indexer gradients' streamed range in two parts
])
def test_tile_backward_vs_oracle(swv, B, T, H, IH, ID, K, o_dtype, exact):
    """The tensor-core backward on the selection of the library's own indexer, against the oracle's
    backward on the same lists: fp32-grade agreement (its factors carry 24 bits), the same tolerance as the
    CUDA-core kernels."""
    g = torch.Generator().manual_seed(T + K)
    bf = torch.bfloat16
    q = (torch.randn(B, T, H, 64, generator=g) / 8).to(bf).to(DEV).transpose(1, 2)
    k, v = (torch.randn(B, T, H, 64, generator=g).to(bf).to(DEV).transpose(1, 2) for _ in range(2))
    qi, ki = ((torch.randn(B, T, IH, ID, generator=g) / ID ** 0.5).to(bf).to(DEV) for _ in range(2))
    w = torch.randn(IH, generator=g).to(DEV)
    d_out = torch.randn(B, T, H, 64, generator=g)
    d_out = (d_out.to(bf) if exact else d_out).to(o_dtype).to(DEV).transpose(1, 2)
    o, idx, valid, scores, sel = swv.ops._dsa_forward(q, k, v, qi, ki, w, K, out_dtype=o_dtype)
    got = swv.ops.dsa_module_bwd(d_out, q, k, v, o, qi, ki, w, idx, valid, scores, sel[0])
    swv.check_status(DEV)
    c = lambda x: x.detach().float().cpu()
    dw_ref = torch.zeros(IH)
    for b in range(B):
        rw = c(scores)[b] * c(valid)[b]
        rq, rk, rv, rrw = O.dsa_attention_bwd(c(d_out)[b], c(q)[b], c(k)[b], c(v)[b], c(o)[b], idx[b].cpu(), c(valid)[b], rw)
        rqi, rki, rdw = O.indexer_bwd(rrw * c(valid)[b], c(qi)[b], c(ki)[b], c(w), idx[b].cpu(), c(valid)[b])
        for x, r in zip(got, (rq, rk, rv, rqi, rki)):
            assert _close(x[b], r)
        dw_ref += rdw
    assert _close(got[5], dw_ref, rel=1e-3)


def test_tile_backward_long_sums_keep_fp32(swv):
    """Gradients of a few queries over a long key range (128 tiles of the sweep) against fp64: the sums must not
    lose bits with their length.  Bound 2^-19 in the 2-norm: every factor is good to about 2^-22 (the
    approximate exponential, the products' fp32 sums) and rounded sums of independent terms do not grow;
    accumulating the whole row in the tensor cores (which truncate at every step) gave 9e-6."""
    T, K, R = 8192, 512, 8
    g = torch.Generator(device=DEV).manual_seed(5)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device=DEV) * scale).to(torch.bfloat16)
    q, k, v = rnd(1, 1, T, 64, scale=0.125), rnd(1, 1, T, 64), rnd(1, 1, T, 64)
    qi, ki = rnd(1, T, 4, 32, scale=32 ** -0.5), rnd(1, T, 4, 32, scale=32 ** -0.5)
    w = torch.randn(4, generator=g, device=DEV)
    d_out = torch.zeros(1, 1, T, 64, dtype=torch.bfloat16, device=DEV)
    d_out[:, :, :R] = rnd(1, 1, R, 64)
    o, idx, valid, scores, sel = swv.ops._dsa_forward(q, k, v, qi, ki, w, K)
    got = swv.ops.dsa_module_bwd(d_out, q, k, v, o, qi, ki, w, idx, valid, scores, sel[0])
    swv.check_status(DEV)
    f = lambda x: x.double()
    ii = idx[0, :R].long()
    rw = f(scores[0, :R] * valid[0, :R])
    kk, vv, dd = f(k[0, 0])[ii], f(v[0, 0])[ii], f(d_out[0, 0, :R])
    e = torch.softmax(torch.einsum("nd,nkd->nk", f(q[0, 0, :R]), kk) / 8, dim=1)
    sm = e / (e * rw).sum(1, keepdim=True)
    drw = sm * (torch.einsum("nd,nkd->nk", dd, vv) - (dd * f(o[0, 0, :R])).sum(1, keepdim=True))
    dq = torch.einsum("nk,nkd->nd", rw * drw, kk) / 8
    dqi = torch.einsum("nk,nkhd->nhd", drw, f(ki[0])[ii]) * f(w)[None, :, None]
    for name, x, r in (("dq", got[0][0, 0, :R], dq), ("dq_idx", got[3][0, :R], dqi)):
        err = float((f(x) - r).norm() / r.norm())
        assert err < 2.0 ** -19, (name, err)


@pytest.mark.parametrize("T,K", [(1024, 512), (3001, 512)])
def test_tile_backward_is_as_exact_as_the_lists(swv, T, K):
    """Both forms of the module backward against fp64 on the same lists: the tensor cores truncate each
    accumulation, which must not cost the tiles more than the CUDA-core kernels' rounded sums lose."""
    H, ID = 2, 64
    g = torch.Generator(device=DEV).manual_seed(T)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device=DEV) * scale).to(torch.bfloat16)
    q, k, v, do = (rnd(1, H, T, 64, scale=x) for x in (0.125, 1.0, 1.0, 1.0))
    qi, ki = rnd(1, T, 4, ID, scale=ID ** -0.5), rnd(1, T, 4, ID, scale=ID ** -0.5)
    w = torch.randn(4, generator=g, device=DEV)
    o, idx, valid, scores, sel = swv.ops._dsa_forward(q, k, v, qi, ki, w, K)
    tiles = swv.ops.dsa_module_bwd(do, q, k, v, o, qi, ki, w, idx, valid, scores, sel[0])
    dq, dk, dv, drw = swv.ops.dsa_attention_bwd(do, q, k, v, o, idx, valid, scores * valid)
    lists = (dq, dk, dv) + swv.ops.dsa_indexer_bwd(drw, qi, ki, w, idx, valid)
    swv.check_status(DEV)
    f = lambda x: x[0].double()
    rw = torch.zeros(T, T, dtype=torch.float64, device=DEV).scatter_(1, idx[0].long(), f(scores))
    mem = torch.zeros(T, T, dtype=torch.bool, device=DEV).scatter_(1, idx[0].long(), True)
    logit = (f(q) @ f(k).transpose(1, 2) / 8).masked_fill(~mem, float("-inf"))
    e = torch.exp(logit - logit.max(-1, keepdim=True).values)
    sm = e / (e * rw).sum(-1, keepdim=True).clamp_min(1e-6)
    gr = sm * (f(do) @ f(v).transpose(1, 2) - (f(do) * f(o)).sum(-1, keepdim=True))
    dg = gr.sum(0)
    dqi = (dg @ f(ki).reshape(T, -1)).reshape(T, 4, ID)
    ref = [(rw * gr) @ f(k) / 8, (rw * gr).transpose(1, 2) @ f(q) / 8, (sm * rw).transpose(1, 2) @ f(do),
           dqi * w.double()[:, None], (dg.T @ f(qi).reshape(T, -1)).reshape(T, 4, ID) * w.double()[:, None]]
    for name, a, b, r in zip(("dq", "dk", "dv", "dq_idx", "dk_idx"), tiles, lists, ref):
        ea, eb = (float((f(x) - r).norm() / r.norm()) for x in (a, b))
        assert ea <= eb, (name, ea, eb)


@pytest.mark.parametrize("B,T,K", [(1, 100, 7), (3, 131, 40), (1, 4097, 300), (2, 4500, 20)])
def test_tile_backward_rebuilds_the_bitmask(swv, B, T, K):
    """Without the bitmask of the forward the backward builds it from the lists: the same gradients bit for bit
    (dw is summed in arrival order).  Rows of several batches in one CTA, a list that ends inside a group of
    32 slots, lists over more than one window of 32 key tiles with empty tiles between."""
    g = torch.Generator().manual_seed(T)
    bf = torch.bfloat16
    q, k, v, do = (torch.randn(B, 1, T, 64, generator=g).to(bf).to(DEV) for _ in range(4))
    qi, ki = (torch.randn(B, T, 4, 32, generator=g).to(bf).to(DEV) for _ in range(2))
    w = torch.randn(4, generator=g).to(DEV)
    o, idx, valid, scores, sel = swv.ops._dsa_forward(q, k, v, qi, ki, w, K)
    args = (do, q, k, v, o, qi, ki, w, idx, valid, scores)
    with_mask, without = swv.ops.dsa_module_bwd(*args, sel[0]), swv.ops.dsa_module_bwd(*args)
    swv.check_status(DEV)
    for name, a, b in zip(("dq", "dk", "dv", "dq_idx", "dk_idx"), with_mask, without):
        assert torch.equal(a, b), name
    assert _close(without[5], with_mask[5].cpu())


def test_module_backward_form_and_memory(swv, monkeypatch):
    """The module takes the tiles for dense selections and the two list kernels for sparse ones, and keeps nothing
    of the size of the bitmask (T^2 / 8 bytes) from its forward to its backward."""
    calls, real = [], swv.ops.dsa_module_bwd
    monkeypatch.setattr(swv.ops, "dsa_module_bwd", lambda *a, **kw: calls.append(1) or real(*a, **kw))
    T, grads = 3000, {}
    for K in (256, 64):
        torch.manual_seed(0)
        m = swv.DeepSeekSparseAttention(d_model=64, attention_heads=1, indexer_heads=4, indexer_dim=32, top_k=K).to(DEV)
        x = torch.randn(1, T, 64, generator=torch.Generator().manual_seed(1)).to(DEV)
        kept = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.append(t) or t, lambda t: t):
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = m(x)
        n = len(calls)
        y.float().square().mean().backward()
        swv.check_status(DEV)
        assert (len(calls) > n) == (K == 256)
        assert [tuple(t.shape) for t in kept if t.dtype == torch.int32] == [(1, T, K)]
        assert all(torch.isfinite(p.grad).all() for p in m.parameters())


def test_tile_backward_in_head_groups(swv):
    """More heads than the room for their list gradients holds (1 GiB: three heads of 8200 tokens with 8192 slots):
    every head's gradients are those of a call with fewer heads, bit for bit, and the indexer's follow the sum
    over all heads, which goes on in the same order (2^-20: the one-group calls are added in another)."""
    T, K, H = 8200, 8192, 5
    g = torch.Generator(device=DEV).manual_seed(3)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device=DEV) * scale).to(torch.bfloat16)
    q, k, v, do = (rnd(1, H, T, 64, scale=x) for x in (0.125, 1.0, 1.0, 1.0))
    qi, ki = rnd(1, T, 2, 32, scale=0.18), rnd(1, T, 2, 32, scale=0.18)
    w = torch.randn(2, generator=g, device=DEV)
    o, idx, valid, scores, _ = swv.ops._dsa_forward(q, k, v, qi, ki, w, K)
    run = lambda h: swv.ops.dsa_module_bwd(*(x[:, h] for x in (do, q, k, v, o)), qi, ki, w, idx, valid, scores)
    every, parts = run(slice(0, H)), (run(slice(0, 3)), run(slice(3, H)))
    swv.check_status(DEV)
    for i in range(3):
        assert torch.equal(every[i], torch.cat([p[i] for p in parts], dim=1))
    for i in (3, 4):
        assert _close(every[i], (parts[0][i] + parts[1][i]).cpu(), rel=2.0 ** -20)


def test_tile_backward_with_a_nan_query(swv):
    """One NaN query (its lists and weights are finite): its gradient and those of the keys it selected are NaN,
    the other queries' gradients are what they are without it, and no wait runs out."""
    T, K, H = 700, 64, 2
    g = torch.Generator().manual_seed(2)
    bf = torch.bfloat16
    q, k, v, do = (torch.randn(1, H, T, 64, generator=g).to(bf).to(DEV) for _ in range(4))
    qi, ki = (torch.randn(1, T, 4, 32, generator=g).to(bf).to(DEV) for _ in range(2))
    w = torch.randn(4, generator=g).to(DEV)
    o, idx, valid, scores, _ = swv.ops._dsa_forward(q, k, v, qi, ki, w, K)
    run = lambda q, o: swv.ops.dsa_module_bwd(do, q, k, v, o, qi, ki, w, idx, valid, scores)
    clean = run(q, o)
    q, o = q.clone(), o.clone()
    q[0, 1, 5], o[0, 1, 5] = float("nan"), float("nan")
    got = run(q, o)
    swv.check_status(DEV)
    assert bool(got[0][0, 1, 5].isnan().all())
    keep = torch.ones(1, H, T, dtype=torch.bool, device=DEV)
    keep[0, 1, 5] = False
    assert torch.equal(got[0][keep], clean[0][keep])
    sel = idx[0, 5].long()
    assert bool(got[1][0, 1, sel].isnan().all()) and bool(got[2][0, 1, sel].isnan().all())
    assert torch.equal(got[1][0, 0], clean[1][0, 0]) and torch.equal(got[2][0, 0], clean[2][0, 0])
