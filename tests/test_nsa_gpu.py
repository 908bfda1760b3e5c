"""NSA-style attention (compressed / selected / sliding-window + gate) against the library-defined
CPU oracle (parity unpinned: the reference has no NSA code)."""
import math

import pytest
import torch

from oracle import nsa as N

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("T,Hq,Hkv,D,topk,window", [(700, 4, 2, 128, 4, 128), (1500, 8, 2, 64, 16, 512),
                                                    (300, 2, 1, 128, 16, 64), (1111, 8, 1, 128, 8, 256),
                                                    (900, 16, 2, 64, 4, 128)])
def test_nsa_vs_oracle(T, Hq, Hkv, D, topk, window):
    import sparse_wsi_vit_b200 as swv
    from sparse_wsi_vit_b200.nsa import nsa_attention
    g = torch.Generator().manual_seed(T)
    q = (torch.randn(1, Hq, T, D, generator=g)).to(torch.bfloat16)
    k = torch.randn(1, Hkv, T, D, generator=g).to(torch.bfloat16)
    v = torch.randn(1, Hkv, T, D, generator=g).to(torch.bfloat16)
    gate = torch.randn(1, T, Hq, 3, generator=g)
    out, o_cmp, o_sel, o_win, blocks = nsa_attention(q.to(DEV), k.to(DEV), v.to(DEV), gate.to(DEV), sel_topk=topk,
                                                     window=window, out_dtype=torch.float32, return_parts=True)
    swv.check_status(DEV)
    ref, r_cmp, r_sel, r_win, r_blocks, margin = N.nsa_attention(q[0], k[0], v[0], gate[0], sel_topk=topk,
                                                                window=window, return_parts=True,
                                                                pooled_dtype=torch.bfloat16)
    _compare(Hq, Hkv, out[0].cpu(), o_cmp[0].cpu(), o_sel[0].cpu(), o_win[0].cpu(), blocks[0].cpu(), ref, r_cmp, r_sel,
             r_win, r_blocks, margin)


def _compare(Hq, Hkv, out, o_cmp, o_sel, o_win, blocks, ref, r_cmp, r_sel, r_win, r_blocks, margin):
    """The oracle pools from the same bf16-rounded values as the library, so the block importances
    agree to fp32 round-off: the selected blocks must be IDENTICAL on every row whose last selected
    and first rejected importance differ by more than 1e-5 relative (ten times the fp32 round-off of the sums) (a smaller gap is a near-tie
    that another summation order may legitimately break the other way), and such near-tie rows
    must be rare."""
    tol = dict(atol=3e-2, rtol=0)
    assert torch.allclose(o_cmp, r_cmp, **tol)
    assert torch.allclose(o_win, r_win, **tol)
    same = (blocks.long() == r_blocks).all(dim=-1)                     # (Hkv, R)
    clear = margin > 1e-5
    assert bool(same[clear].all()), f"{int((~same & clear).sum())} rows with a clear margin selected other blocks"
    assert clear.float().mean() > 0.9
    rows = same.repeat_interleave(Hq // Hkv, dim=0)                    # (Hq, R)
    assert (o_sel - r_sel)[rows].abs().max() < 3e-2
    assert (out - ref)[rows].abs().max() < 3e-2
    assert (out - ref)[rows].abs().mean() < 2e-3


def test_nsa_benchmark_size_sampled_rows():
    """65536 tokens, 16 query / 2 kv heads, head_dim 128, 32/16 compression, 16 blocks of 64, window
    512 (the NSA configuration that is timed): full GPU run, oracle on 96 sampled query rows
    against all keys."""
    import sparse_wsi_vit_b200 as swv
    from sparse_wsi_vit_b200.nsa import nsa_attention
    T, Hq, Hkv, D = 65536, 16, 2, 128
    g = torch.Generator().manual_seed(65)
    q = torch.randn(1, Hq, T, D, generator=g).to(torch.bfloat16)
    k = torch.randn(1, Hkv, T, D, generator=g).to(torch.bfloat16)
    v = torch.randn(1, Hkv, T, D, generator=g).to(torch.bfloat16)
    gate = torch.randn(1, T, Hq, 3, generator=g)
    rows = torch.cat([torch.arange(0, 16), torch.randperm(T, generator=g)[:64].sort().values, torch.arange(T - 16, T)])
    out, o_cmp, o_sel, o_win, blocks = nsa_attention(q.to(DEV), k.to(DEV), v.to(DEV), gate.to(DEV),
                                                     out_dtype=torch.float32, return_parts=True)
    one = nsa_attention(q.to(DEV), k.to(DEV), v.to(DEV), gate.to(DEV), out_dtype=torch.float32)
    swv.check_status(DEV)
    assert (one - out).abs().max() < 1e-5
    ref, r_cmp, r_sel, r_win, r_blocks, margin = N.nsa_attention(q[0], k[0], v[0], gate[0], return_parts=True,
                                                                rows=rows, pooled_dtype=torch.bfloat16)
    _compare(Hq, Hkv, out[0, :, rows].cpu(), o_cmp[0, :, rows].cpu(), o_sel[0, :, rows].cpu(), o_win[0, :, rows].cpu(),
             blocks[0][:, rows].cpu(), ref, r_cmp, r_sel, r_win, r_blocks, margin)


def test_nsa_single_call_equals_stepwise():
    """`swv_nsa_attn_fwd` (one call, device-built block lists, caller workspace, gates applied in the
    branch epilogues) against the step-by-step composition (branch outputs + gate kernel)."""
    import sparse_wsi_vit_b200 as swv
    from sparse_wsi_vit_b200.nsa import nsa_attention
    T, Hq, Hkv, D = 1100, 8, 2, 128
    g = torch.Generator().manual_seed(5)
    q = torch.randn(1, Hq, T, D, generator=g).to(torch.bfloat16).to(DEV)
    k = torch.randn(1, Hkv, T, D, generator=g).to(torch.bfloat16).to(DEV)
    v = torch.randn(1, Hkv, T, D, generator=g).to(torch.bfloat16).to(DEV)
    gate = torch.randn(1, T, Hq, 3, generator=g).to(DEV)
    one = nsa_attention(q, k, v, gate, sel_topk=8, window=256, out_dtype=torch.float32)
    parts = nsa_attention(q, k, v, gate, sel_topk=8, window=256, out_dtype=torch.float32, return_parts=True)
    swv.check_status(DEV)
    # same kernels and the same order of additions; the fused epilogues contract g * o + acc into one
    # FMA where the stand-alone gate kernel may round the product first
    assert (one - parts[0]).abs().max() < 1e-5


@pytest.mark.parametrize("T", [300, 6000, 17000, 66000])
def test_selection_on_plateaus_takes_the_lowest_blocks(T):
    """Zero queries: every compressed token is equally important, so all full blocks tie and the lowest
    indices must be taken.  More ties than the short selection's candidate buffer holds (its arg-max
    fallback), the two register sizes of the short form, and more blocks than it takes."""
    import sparse_wsi_vit_b200 as swv
    from sparse_wsi_vit_b200.nsa import nsa_attention
    g = torch.Generator().manual_seed(T)
    q = torch.zeros(1, 2, T, 64, dtype=torch.bfloat16, device=DEV)
    k, v = (torch.randn(1, 1, T, 64, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    gate = torch.zeros(1, T, 2, 3, device=DEV)
    _, _, o_sel, _, blocks = nsa_attention(q, k, v, gate, window=128, return_parts=True)
    swv.check_status(DEV)
    n = min(16, -(-T // 64))
    assert bool((blocks[0, 0] == torch.arange(n, device=DEV)).all())
    # equal scores: the selected branch is the mean of the selected values; P is 1 before normalisation,
    # so only the bf16 rounding of the inputs and the fp32 sums are left
    mean = v[0, 0, :min(T, n * 64)].float().mean(0)
    assert (o_sel[0] - mean).abs().max() < 1e-4


@pytest.mark.parametrize("D", [64, 128])
def test_selected_branch_dominant_key_is_not_rounded(D):
    """Two keys per query carry all the weight: one in the first selected block, a larger one (by x = 0.3 .. 5
    in the log2 domain) in the last.  P is rounded to bf16 relative to the row's maximum, so the larger key's
    probability is exactly 1 and only the smaller one's rounding (2^-9 of it) is left, beside the 2^-22 of the
    approximate exponential and the fp32 sums: |error| <= 2^-9 w_small |v_small| + 2^-18 max|v|, w = its weight."""
    from sparse_wsi_vit_b200.nsa import selected_attention
    R, blk = 64, 64
    T = 4 * blk
    g = torch.Generator().manual_seed(D)
    k = torch.zeros(1, 1, T, D)
    k[..., 0] = -64.0                                     # every other key: weight 2^-60 and less
    k[0, 0, 3] = 0.0
    k[0, 0, 3, 1] = 1.0                                   # logit of the small key: channel 1 of the query
    k[0, 0, 200] = 0.0
    k[0, 0, 200, 2] = 1.0                                 # of the large key: channel 2
    x = torch.linspace(0.3, 5.0, R) * D ** 0.5 * math.log(2.0)
    q = torch.zeros(1, 1, R, D)
    q[..., 0], q[0, 0, :, 2] = D ** 0.5, x
    q, k = q.to(torch.bfloat16), k.to(torch.bfloat16)
    v = torch.randn(1, 1, T, D, generator=g).to(torch.bfloat16)
    blocks = torch.tensor([0, 1, 3], dtype=torch.int32).repeat(R, 1)[None, None]
    o = selected_attention(q.to(DEV), k.to(DEV), v.to(DEV), blocks.to(DEV), blk)[0, 0].cpu().double()
    keys = torch.cat([torch.arange(b * blk, (b + 1) * blk) for b in (0, 1, 3)])
    w = torch.softmax(q[0, 0].double() @ k[0, 0, keys].double().T / D ** 0.5, dim=1)
    vd = v[0, 0].double()
    bound = 2.0 ** -9 * w[:, 3:4] * vd[3].abs() + 2.0 ** -18 * vd.abs().max()
    assert bool(((o - w @ vd[keys]).abs() <= bound).all())


@pytest.mark.parametrize("T,topk", [(3000, 16), (16384, 16), (4000, 40), (66000, 16)])
def test_selection_with_nan_rows_lists_valid_blocks(T, topk):
    """A NaN query (its own row) and a NaN key (every row): NaN importances count as 0, so each row still lists
    k_eff ascending blocks of the sequence, the lowest ones of a row without any other importance.  Block counts
    with and without padding entries in the short form's registers, and both ways to the arg-max loop."""
    import sparse_wsi_vit_b200 as swv
    from sparse_wsi_vit_b200.nsa import nsa_attention
    g = torch.Generator().manual_seed(T)
    q, k, v = (torch.randn(1, h, T, 64, generator=g).to(torch.bfloat16).to(DEV) for h in (2, 1, 1))
    gate = torch.zeros(1, T, 2, 3, device=DEV)
    n = -(-T // 64)
    run = lambda q, k: nsa_attention(q, k, v, gate, sel_topk=topk, window=128, return_parts=True)
    blocks = run(q, k)[4]
    q1 = q.clone()
    q1[:, :, 7] = float("nan")
    got, lowest = run(q1, k), torch.arange(min(topk, n), device=DEV)
    assert torch.equal(got[4][0, 0, 7], lowest.int()) and bool(got[2][0, :, 7].isnan().all())
    keep = torch.arange(T, device=DEV) != 7
    assert torch.equal(got[4][:, :, keep], blocks[:, :, keep])
    k1 = k.clone()
    k1[:, :, T // 2] = float("nan")
    b = run(q, k1)[4]
    swv.check_status(DEV)
    assert bool((b[..., 1:] > b[..., :-1]).all()) and int(b.min()) >= 0 and int(b.max()) < n


@pytest.mark.parametrize("aligned", [True, False])
def test_selected_branch_ignores_blocks_outside_the_keys(aligned):
    """Block indices below 0 and behind the last block attend nothing and nothing is read through them, on
    tensor-core tiles and (odd query strides) on CUDA cores."""
    from sparse_wsi_vit_b200.nsa import selected_attention
    T, D = 300, 64
    g = torch.Generator().manual_seed(8)
    q = torch.randn(1, 4, T, D + 1, generator=g).to(torch.bfloat16).to(DEV)[..., :D]
    k, v = (torch.randn(1, 2, T, D, generator=g).to(torch.bfloat16).to(DEV) for _ in range(2))
    q = q.contiguous() if aligned else q
    run = lambda blocks: selected_attention(q, k, v, torch.tensor(blocks, dtype=torch.int32, device=DEV).repeat(2, T, 1)[None], 64)
    want = run([1, 4])
    assert torch.isfinite(want).all()
    for blocks in ([1, 4, -1, 5, -2 ** 31, 2 ** 31 - 1], [-7, 1, 9, 4, 6, 2 ** 30]):
        assert torch.equal(run(blocks), want)
