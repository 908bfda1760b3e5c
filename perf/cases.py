"""The work this library is used for, as a list of measurable cases.

Slide encoders run on bags of patch embeddings whose size varies from slide to slide: a biopsy has a
few hundred to a few thousand patches, a resection up to about 10^5.  The cases cover what a user's
program calls: whole encoders in inference, a training pass through the attention layer and through
an encoder, the single attention operators at the sizes this repository's benchmark configures them
with, and the static / 2-D block-pattern / NSA attention that the same package offers.

Every case is a dict of plain values; ``prepare`` makes on the GPU what a program holds before the
call, ``run`` is one pass through the public entry points.
"""
import math

import torch

import sparse_wsi_vit_b200 as swv
from sparse_wsi_vit_b200.nsa import nsa_attention
from sparse_wsi_vit_b200.training import slide_step

PATCH = 224.0          # pixels between neighbouring patches, the unit of the slide coordinates
GRID = 512             # patches per side of the slide grid the tissue cells are drawn from
FEATURES = 1280        # width of a patch embedding

# encoder sizes: the constructor's defaults, and the 12-layer model of the ragged-batch benchmark
MODELS = {
    "default": dict(embed_dim=384, num_heads=6, num_layers=6, indexer_heads=4, indexer_dim=32, top_k=512),
    "large": dict(embed_dim=768, num_heads=12, num_layers=12, indexer_heads=4, indexer_dim=64, top_k=2048),
}


def listed():
    return [
        # Inference on a small biopsy with the default encoder: latency and launches count.
        dict(name="encoder_biopsy", kind="encoder", model="default", patches=1021, rope=False),
        # Inference on the smallest slide of the ragged batch, 12 layers with 2-D RoPE: the large model.
        dict(name="encoder_slide_24k", kind="encoder", model="large", patches=24576, rope=True),
        # One DSA layer at 16384 tokens, top-2048: one key in 8 selected (the dense sweep).
        dict(name="dsa_layer_16k", kind="dsa", tokens=16384, shard=1, heads=8, indexer_dim=64, top_k=2048),
        # One DSA layer at 65536 tokens, top-2048: the headline configuration (one key in 32).
        dict(name="dsa_layer_64k", kind="dsa", tokens=65536, shard=1, heads=8, indexer_dim=64, top_k=2048),
        # The reference-shaped operators in fp32 (no autocast), an odd size.
        dict(name="dsa_ops_f32", kind="dsa_f32", tokens=4099, heads=6, indexer_dim=32, top_k=512),
        # Forward and backward of one DSA layer at the benchmark's size, bf16 autocast.
        dict(name="train_layer_16k", kind="train_layer", tokens=16384, heads=8, indexer_dim=64, top_k=2048),
        # A training pass (forward, loss, backward) of a 2-layer default-width encoder on an ordinary slide.
        dict(name="train_encoder", kind="train_encoder", patches=6007, top_k=512),
        # The block-sparse sweep's middle: 32768 tokens, 16 x 128, block 128, band +-2 + global + 5 % extra blocks.
        dict(name="block_sparse_32k", kind="block_sparse", tokens=32768, heads=16, head_dim=128, block=128, p=0.05),
        # The 2-layer 2-D block-pattern model, 4096 patches on a 64 x 64 grid.
        dict(name="grid2d_4096", kind="grid2d", tiles=8),
        # One NSA layer at 65536 tokens, 16 query / 2 kv heads.
        dict(name="nsa_64k", kind="nsa", tokens=65536, heads=16, kv_heads=2, head_dim=128),
        # The same layer on a small slide of odd size.
        dict(name="nsa_5k", kind="nsa", tokens=5003, heads=16, kv_heads=2, head_dim=128),
        # The static-pattern encoder (2 layers, window 3) under autocast.
        dict(name="static_4096", kind="static", patches=4096, window=3, dilation=1, autocast=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["encoder", "encoder", "dsa", "dsa", "dsa_f32", "train_layer", "train_encoder", "block_sparse",
                       "grid2d", "nsa", "static"])
    if kind == "encoder":
        model = rng.choice(["default", "default", "large"])
        return dict(kind=kind, model=model, patches=_log_int(rng, 256, 24576), rope=rng.random() < 0.5)
    if kind == "dsa":           # shard > 1: one rank's queries against all keys of a sequence-sharded slide
        return dict(kind=kind, tokens=_log_int(rng, 256, 65536), shard=rng.choice([1, 1, 1, 2, 8]),
                    heads=rng.choice([6, 8, 12]), indexer_dim=rng.choice([32, 64]), top_k=rng.choice([512, 1024, 2048]))
    if kind == "dsa_f32":
        return dict(kind=kind, tokens=_log_int(rng, 256, 8192), heads=rng.choice([6, 8]), indexer_dim=rng.choice([32, 64]),
                    top_k=rng.choice([256, 512]))
    if kind == "train_layer":
        return dict(kind=kind, tokens=_log_int(rng, 1024, 16384), heads=rng.choice([6, 8]), indexer_dim=rng.choice([32, 64]),
                    top_k=rng.choice([512, 1024, 2048]))
    if kind == "train_encoder":
        return dict(kind=kind, patches=_log_int(rng, 512, 12288), top_k=rng.choice([256, 512, 1024]))
    if kind == "block_sparse":
        return dict(kind=kind, tokens=_log_int(rng, 2048, 65536), heads=rng.choice([8, 12, 16]),
                    head_dim=rng.choice([64, 128]), block=rng.choice([64, 128]), p=rng.choice([0.0, 0.01, 0.05, 0.25]))
    if kind == "grid2d":
        return dict(kind=kind, tiles=rng.randint(4, 28))
    if kind == "nsa":
        return dict(kind=kind, tokens=_log_int(rng, 1024, 65536), heads=rng.choice([8, 16]), kv_heads=2,
                    head_dim=rng.choice([64, 128]))
    return dict(kind=kind, patches=_log_int(rng, 512, 32768), window=rng.choice([1, 3, 16, 64]),
                dilation=rng.choice([1, 1, 2]), autocast=rng.random() < 0.7)


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _module(cls, seed, **kw):
    torch.manual_seed(seed)
    with torch.device("cuda"):
        return cls(**kw)


def _coords(g, n):
    """n tissue cells of the slide grid in raster order, in pixels."""
    cells = torch.randperm(GRID * GRID, generator=g, device="cuda")[:n].sort().values
    return torch.stack([cells // GRID, cells % GRID], dim=1).float() * PATCH


def _dsa_tensors(case, g, dtype):
    """q, k, v ~ N(0,1) (q scaled by 1/sqrt(64)), indexer projections N(0,1/ID), head weights N(0,1)."""
    t, h, i = case["tokens"], case["heads"], case["indexer_dim"]
    tq = -(-t // case.get("shard", 1))
    q = _randn(g, 1, tq, h, 64, scale=0.125, dtype=dtype).transpose(1, 2)
    k, v = (_randn(g, 1, t, h, 64, dtype=dtype).transpose(1, 2) for _ in range(2))
    qi = _randn(g, 1, tq, 4, i, scale=i ** -0.5, dtype=dtype)
    ki = _randn(g, 1, t, 4, i, scale=i ** -0.5, dtype=dtype)
    return q, k, v, qi, ki, _randn(g, 4, dtype=torch.float32)


def _grid_coords(tiles):
    """Block-major tokens: one 8 x 8 spatial tile per block of 64 tokens."""
    t = torch.arange(tiles * tiles * 64, device="cuda")
    blk, tin = t // 64, t % 64
    return torch.stack([(blk // tiles) * 8 + tin // 8, (blk % tiles) * 8 + tin % 8], dim=1).float()


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    s = {"case": case}
    if kind == "encoder":
        n = case["patches"]
        s["net"] = _module(swv.DSAViTSlideEncoder, seed, in_features=FEATURES, out_features=2, num_cls=2,
                           rope_coord_high=PATCH * GRID if case["rope"] else None, **MODELS[case["model"]]).eval()
        s["x"], s["coords"] = _randn(g, n, FEATURES), _coords(g, n)
    elif kind == "dsa":
        s["t"] = _dsa_tensors(case, g, torch.bfloat16)
    elif kind == "dsa_f32":
        s["t"] = _dsa_tensors(case, g, torch.float32)
    elif kind == "train_layer":
        d = case["heads"] * 64
        s["net"] = _module(swv.DeepSeekSparseAttention, seed, d_model=d, attention_heads=case["heads"], indexer_heads=4,
                           indexer_dim=case["indexer_dim"], top_k=case["top_k"])
        s["x"] = _randn(g, 1, case["tokens"], d, dtype=torch.float32).requires_grad_()      # a LayerNorm's output
        s["dy"] = _randn(g, 1, case["tokens"], d)
    elif kind == "train_encoder":
        n = case["patches"]
        s["net"] = _module(swv.DSAViTSlideEncoder, seed, in_features=FEATURES, out_features=2, embed_dim=384, num_heads=6,
                           num_layers=2, num_cls=2, indexer_heads=4, indexer_dim=32, top_k=case["top_k"],
                           rope_coord_high=PATCH * GRID).train()
        s["batch"] = {"input": _randn(g, 1, n, FEATURES), "coords": _coords(g, n)[None],
                      "label": torch.tensor([seed % 2], device="cuda")}
    elif kind == "block_sparse":
        n, h, d, bs = case["tokens"], case["heads"], case["head_dim"], case["block"]
        s["qkv"] = tuple(_randn(g, 1, h, n, d) for _ in range(3))
        lists = swv.patterns.band_random_blocks(-(-n // bs), band=2, n_global=1, p=case["p"], seed=1)
        s["lists"] = tuple(torch.from_numpy(a).cuda() for a in lists)
    elif kind == "grid2d":
        m = case["tiles"]
        s["net"] = _module(swv.BlockSparse2DViTSlideEncoder, seed, in_features=FEATURES, out_features=2, embed_dim=384,
                           num_heads=6, num_layers=2, num_cls=1, block=64, coord_high=8.0 * m).eval()
        s["x"], s["coords"] = _randn(g, m * m * 64, FEATURES, dtype=torch.float32), _grid_coords(m)
        lists = swv.patterns.chebyshev_grid_blocks(m, m, 1, global_blocks=[m * m])
        s["lists"] = tuple(torch.from_numpy(a).cuda() for a in lists)
    elif kind == "nsa":
        n, h, hk, d = case["tokens"], case["heads"], case["kv_heads"], case["head_dim"]
        s["t"] = (_randn(g, 1, h, n, d), _randn(g, 1, hk, n, d), _randn(g, 1, hk, n, d),
                  _randn(g, 1, n, h, 3, dtype=torch.float32))
    else:
        s["net"] = _module(swv.StaticSparseViTSlideEncoder, seed, in_features=FEATURES, out_features=2, embed_dim=384,
                           num_heads=6, num_layers=2, num_cls=1, window_size=case["window"],
                           dilation=case["dilation"]).eval()
        s["x"] = _randn(g, 1, case["patches"], FEATURES, dtype=torch.float32)
    return s


# ------------------------------------------------------------------ one pass
def _grads(net):
    return {n: p.grad for n, p in net.named_parameters()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "encoder":
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return state["net"](state["x"], state["coords"])["logits"]
    if kind == "dsa":
        return swv.dsa_sparse_attention(*state["t"], case["top_k"], return_topk=True)
    if kind == "dsa_f32":
        q, k, v, qi, ki, w = state["t"]
        b, h, t, d = q.shape
        idx, valid, scores = swv.LightningIndexerFunction.apply(qi, ki, w, b, t, 4, qi.shape[3], case["top_k"])
        o = torch.empty_like(q)
        return swv.DSAAttentionFunction.apply(q, k, v, idx, valid, scores * valid, o, b, h, t, d, case["top_k"]), idx
    if kind == "train_layer":
        net, x = state["net"], state["x"]
        net.zero_grad(set_to_none=True)
        x.grad = None
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = net(x)
        y.backward(state["dy"].to(y.dtype))
        return {"y": y, "dx": x.grad, **_grads(net)}
    if kind == "train_encoder":
        net = state["net"]
        net.zero_grad(set_to_none=True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss, _, logits = slide_step(net, state["batch"])
        loss.backward()
        return {"loss": loss, "logits": logits, **_grads(net)}
    if kind == "block_sparse":
        return swv.block_sparse_attention(*state["qkv"], *state["lists"], case["block"])
    if kind == "grid2d":
        with torch.no_grad():
            return state["net"](state["x"], state["coords"], *state["lists"])["logits"]
    if kind == "nsa":
        return nsa_attention(*state["t"])
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16, enabled=case["autocast"]):
        return state["net"](state["x"])["logits"]


# ------------------------------------------------------------------ what a pass cannot do without
def _dsa_flops(tq, tk, heads, indexer_dim, top_k, d=64):
    """Every indexer score once (heads collapsed), and both products of the selected keys."""
    return 2.0 * tq * tk * indexer_dim + 4.0 * tq * min(top_k, tk) * heads * d


def _dsa_bwd_flops(t, heads, indexer_dim, top_k, d=64):
    """Per selected (query, key) pair: five products of the attention, three of the indexer's gradients."""
    return t * min(top_k, t) * (10.0 * heads * d + 6.0 * 4 * indexer_dim)


def _block_flops(e, n, expansion=4):
    """The Linears of one transformer block (QKV, output projection, MLP)."""
    return 2.0 * n * e * e * (4 + 2 * expansion)


def work(case):
    kind = case["kind"]
    if kind in ("encoder", "train_encoder"):
        m = MODELS[case["model"]] if kind == "encoder" else dict(embed_dim=384, num_heads=6, num_layers=2, indexer_heads=4,
                                                                  indexer_dim=32, top_k=case["top_k"])
        n, e, ie = case["patches"] + 2, m["embed_dim"], m["indexer_heads"] * m["indexer_dim"]
        params = FEATURES * e + m["num_layers"] * e * (12 * e + 2 * ie)
        gemm = 2.0 * n * params
        attn = m["num_layers"] * _dsa_flops(n, n, m["num_heads"], m["indexer_dim"], m["top_k"])
        if kind == "encoder":
            return {"bytes": 2.0 * n * FEATURES + 4.0 * params, "flops": gemm + attn}
        bwd = m["num_layers"] * _dsa_bwd_flops(n, m["num_heads"], m["indexer_dim"], m["top_k"])
        return {"bytes": 2.0 * n * FEATURES + 8.0 * params, "flops": 3 * gemm + attn + bwd}
    if kind in ("dsa", "dsa_f32"):
        t, h, i, es = case["tokens"], case["heads"], case["indexer_dim"], 2 if kind == "dsa" else 4
        tq = -(-t // case.get("shard", 1))
        rows = es * ((2 * tq + 2 * t) * h * 64 + (tq + t) * 4 * i)
        lists = tq * case["top_k"] * (12.0 if kind == "dsa" else 4.0)
        return {"bytes": rows + lists, "flops": _dsa_flops(tq, t, h, i, case["top_k"])}
    if kind == "train_layer":
        t, h, i = case["tokens"], case["heads"], case["indexer_dim"]
        e = 64 * h
        params = 4 * e * e + 2 * e * 4 * i
        flops = 6.0 * t * params + _dsa_flops(t, t, h, i, case["top_k"]) + _dsa_bwd_flops(t, h, i, case["top_k"])
        return {"bytes": t * e * (4.0 + 2 + 2 + 4) + 8.0 * params, "flops": flops}
    if kind == "block_sparse":
        n, h, d, bs = case["tokens"], case["heads"], case["head_dim"], case["block"]
        nb = -(-n // bs)
        # band of 5 and one global block, then a share p of the rest
        per_row = min(nb, 6) + case["p"] * max(0, nb - 6)
        return {"bytes": 8.0 * n * h * d, "flops": 4.0 * n * bs * per_row * h * d}
    if kind == "grid2d":
        n, e = case["tiles"] ** 2 * 64 + 1, 384
        flops = 2.0 * n * FEATURES * e + 2 * (_block_flops(e, n) + 4.0 * n * 10 * 64 * e)
        return {"bytes": 4.0 * n * FEATURES + 4.0 * (FEATURES * e + 24 * e * e), "flops": flops}
    if kind == "nsa":
        n, h, hk, d = case["tokens"], case["heads"], case["kv_heads"], case["head_dim"]
        n_c = max(0, (n - 32) // 16 + 1)
        keys = n_c * 1.5 + min(n, 16 * 64) + min(n, 513)      # the block importances need the first product once more
        return {"bytes": n * d * (4.0 * h + 4.0 * hk) + 12.0 * n * h, "flops": 4.0 * n * h * d * keys}
    n, e = case["patches"] + 1, 384
    flops = 2.0 * n * FEATURES * e + 2 * (_block_flops(e, n) + 4.0 * n * (2 * case["window"] + 2) * e)
    return {"bytes": 4.0 * n * FEATURES + 4.0 * (FEATURES * e + 24 * e * e), "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "dsa":                # bf16 outputs; a near-tie of two scores shifts the rest of its row's list
        return {"rel": 1e-2, "differ": 2e-3}
    if kind == "dsa_f32":            # fp32 attention over lists that TF32 scores select and weigh
        return {"rel": 1e-3, "differ": 2e-3}
    if kind in ("block_sparse", "nsa"):
        return {"rel": 1e-2}
    if kind == "static" and not case["autocast"]:
        return {"rel": 1e-4}
    return {"rel": 2e-2}             # several bf16 layers (or their gradients) one after another
