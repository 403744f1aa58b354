"""Performance cases: what a user of the framework has it do, through its public entry points.

Every case is a dict of plain values.  ``listed()`` names twelve of them, ``draw()`` gives more from the same ranges;
``prepare`` / ``run`` / ``work`` / ``tolerance`` / ``exact`` say how one is built, run, counted and checked.

Kinds (the shapes are those of the model presets under ``configs/`` and of ``benchmarks/_common.py``):

``decode``     one new token per sequence through a transformer block with its KV cache (the inner step of ``generate``)
``prefill``    a whole prompt through a block into an empty KV cache (the first call of ``generate``)
``model``      one new token through a whole small model: embedding, all blocks, final norm, head -> logits
``train``      a block's forward and backward; ``flat`` puts its parameters into the flat buffers that training uses,
               ``ac`` recomputes the block in the backward pass (activation checkpointing)
``packed``     the attention layer on a packed sequence with document ids, forward and backward
``loss``       the output head fused with the cross entropy, forward and backward
``moe``        a mixture-of-experts feed-forward layer, forward and backward
``fp8``        a SwiGLU MLP whose weights are tagged for fp8, forward and backward
``adamw``      one AdamW step over the flat buffers of a block
"""

from __future__ import annotations

import math

import torch

DEV = "cuda"
BF = torch.bfloat16
F64 = torch.float64
EPS = 1e-5

# Shapes of the presets: the 125 M benchmark model, moe_small's attention with a dense
# feed-forward of its width, llama_7b and llama_13b
DIMS = {
    "125m": dict(dim=768, heads=12, kv=12, ffn=2048, theta=10000.0),
    "small": dict(dim=2048, heads=16, kv=4, ffn=7168, theta=500000.0),
    "7b": dict(dim=4096, heads=32, kv=8, ffn=14336, theta=500000.0),
    "13b": dict(dim=5120, heads=40, kv=8, ffn=17920, theta=500000.0),
}
MAX_SEQ = 4096


def listed() -> list[dict]:
    return [
        # interactive generation with the 125 M model: one sequence, launches and host work decide
        dict(name="model_125m_b1", kind="model", **DIMS["125m"], layers=12, vocab=32000, batch=1, ctx=300),
        # interactive generation with a 7B model, one block of it
        dict(name="decode_7b_b1", kind="decode", **DIMS["7b"], batch=1, ctx=1000),
        # batched generation with a long context
        dict(name="decode_13b_b16", kind="decode", **DIMS["13b"], batch=16, ctx=2047),
        # prompts of uneven length on their way into the cache
        dict(name="prefill_7b_2x777", kind="prefill", **DIMS["7b"], batch=2, seq=777),
        # the training step's main work at the benchmark's shape (micro-batch 2 x 4096)
        dict(name="train_7b_2x4096", kind="train", **DIMS["7b"], batch=2, seq=4096, flat=True, ac=True),
        # a small model on a ragged batch, as a hand-written loop over plain modules trains it
        dict(name="train_125m_3x333", kind="train", **DIMS["125m"], batch=3, seq=333, flat=False, ac=False),
        # packed documents (data.pack_sequences) in the attention layer
        dict(name="packed_13b_1x3000", kind="packed", **DIMS["13b"], batch=1, seq=3000, docs=7),
        # head and loss over the large vocabulary, with ignored labels
        dict(name="loss_128k_2047", kind="loss", dim=4096, vocab=128256, tokens=2047),
        # moe_small: 8 experts, top-2, one Linear module per expert
        dict(name="moe_8x_2x1024", kind="moe", dim=2048, hidden=7168, experts=8, topk=2, router="softmax_topk",
             packed=False, shared=0, batch=2, seq=1024),
        # fine-grained experts: 64 of 1408, top-6, packed weights and a shared expert
        dict(name="moe_64x_1x1777", kind="moe", dim=2048, hidden=1408, experts=64, topk=6, router="sigmoid_topk",
             packed=True, shared=2, batch=1, seq=1777),
        # fp8 training of the 7B feed-forward
        dict(name="fp8_7b_2000", kind="fp8", dim=4096, ffn=14336, tokens=2000),
        # the optimizer on one 7B block
        dict(name="adamw_7b", kind="adamw", **DIMS["7b"]),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(["model", "decode", "decode", "prefill", "train", "packed", "loss", "moe", "fp8", "adamw"])
    if kind == "model":
        return dict(kind=kind, **DIMS["125m"], layers=rng.randint(4, 12), vocab=32000, batch=_log_int(rng, 1, 8),
                    ctx=_log_int(rng, 16, 2000))
    if kind == "decode":
        return dict(kind=kind, **DIMS[rng.choice(["125m", "small", "7b", "13b"])], batch=_log_int(rng, 1, 32),
                    ctx=_log_int(rng, 16, 4000))
    if kind == "prefill":
        return dict(kind=kind, **DIMS[rng.choice(["125m", "small", "7b", "13b"])], batch=rng.randint(1, 3),
                    seq=_log_int(rng, 9, 1500))
    if kind == "train":
        flat = rng.random() < 0.5
        return dict(kind=kind, **DIMS[rng.choice(["125m", "small", "7b"])], batch=rng.randint(1, 4),
                    seq=_log_int(rng, 100, 2048), flat=flat, ac=flat and rng.random() < 0.5)
    if kind == "packed":
        return dict(kind=kind, **DIMS[rng.choice(["125m", "small", "7b", "13b"])], batch=rng.randint(1, 2),
                    seq=_log_int(rng, 200, 4096), docs=rng.randint(1, 20))
    if kind == "loss":
        dim, vocab = rng.choice([(768, 32000), (2048, 128256), (4096, 128256), (2048, 102400)])
        return dict(kind=kind, dim=dim, vocab=vocab, tokens=_log_int(rng, 100, 2500))
    if kind == "moe":
        if rng.random() < 0.5:
            shape = dict(dim=2048, hidden=7168, experts=8, topk=2, router="softmax_topk", packed=rng.random() < 0.5)
        else:
            shape = dict(dim=2048, hidden=1408, experts=64, topk=6, router="sigmoid_topk", packed=True)
        return dict(kind=kind, **shape, shared=rng.choice([0, 1]), batch=rng.randint(1, 2),
                    seq=_log_int(rng, 128, 2048))
    if kind == "fp8":
        dim, ffn = rng.choice([(2048, 7168), (4096, 14336), (5120, 17920)])
        return dict(kind=kind, dim=dim, ffn=ffn, tokens=16 * _log_int(rng, 8, 256))
    shape = dict(DIMS[rng.choice(["125m", "small", "7b"])])
    shape["ffn"] = 64 * rng.randint(shape["ffn"] // 128, shape["ffn"] // 64)
    return dict(kind=kind, **shape)


# --------------------------------------------------------------------------- inputs
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _normal(g, *shape, std=1.0, dtype=BF):
    return torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=g)


def _fill(module, g, std=0.02) -> None:
    """Weights of a trained net's size: matrices N(0, std), gains around one."""
    with torch.no_grad():
        for p in module.parameters():
            p.normal_(0.0, std, generator=g) if p.dim() > 1 else p.normal_(1.0, 0.1, generator=g)


def _build(make):
    with torch.device(DEV):
        old = torch.get_default_dtype()
        torch.set_default_dtype(BF)
        try:
            return make()
        finally:
            torch.set_default_dtype(old)


def _config(c, **over):
    from kempnerforge_b200.config import ModelConfig

    base = dict(dim=c["dim"], n_layers=1, n_heads=c["heads"], n_kv_heads=c["kv"], vocab_size=c.get("vocab", 1024),
                ffn_hidden_dim=c["ffn"], max_seq_len=MAX_SEQ, rope_theta=c["theta"])
    base.update(over)
    return ModelConfig(**base)


def _rope(c):
    from kempnerforge_b200.models.position import precompute_rope_frequencies

    return precompute_rope_frequencies(c["dim"] // c["heads"], MAX_SEQ, c["theta"], device=DEV)


def _doc_ids(c, seed):
    g = torch.Generator().manual_seed(int(seed) + 1)
    rows = []
    for _ in range(c["batch"]):
        cuts = torch.randint(1, c["seq"], (c["docs"] - 1,), generator=g) if c["docs"] > 1 else torch.empty(0, dtype=torch.long)
        ids = torch.zeros(c["seq"], dtype=torch.long)
        ids[cuts] = 1
        rows.append(ids.cumsum(0))
    return torch.stack(rows).to(DEV)


def prepare(case: dict, seed: int):
    c, g = dict(case), _gen(seed)
    kind = c["kind"]
    s = {"c": c}
    hd = c["dim"] // c["heads"] if "heads" in c else 0
    if kind in ("decode", "prefill", "train"):
        from kempnerforge_b200.models.transformer import TransformerBlock

        block = _build(lambda: TransformerBlock(_config(c), 0))
        _fill(block, g)
        s["block"] = block
        s["cos"], s["sin"] = _rope(c)
    if kind in ("decode", "prefill"):
        from kempnerforge_b200.models.attention import KVCache

        block.eval()
        room = min(MAX_SEQ, c.get("ctx", c.get("seq", 0)) + 64)   # the prompt and what generate() may still add
        cache = KVCache(c["batch"], room, c["kv"], hd, BF, torch.device(DEV))
        if kind == "decode":
            cache.k[:, : c["ctx"]].normal_(0.0, 1.0, generator=g)
            cache.v[:, : c["ctx"]].normal_(0.0, 1.0, generator=g)
        s["cache"] = cache
        s["x"] = _normal(g, c["batch"], c.get("seq", 1), c["dim"])
    elif kind == "train":
        if c["flat"]:
            from kempnerforge_b200.parallel.flat import FlatParamGroup

            s["flat"] = FlatParamGroup("layers.0", block.named_parameters())
        block.ac_mode = "full" if c["ac"] else "none"
        block.train()
        s["x"] = _normal(g, c["batch"], c["seq"], c["dim"]).requires_grad_(True)
        s["dy"] = _normal(g, c["batch"], c["seq"], c["dim"], std=0.01)
    elif kind == "model":
        from kempnerforge_b200.models.attention import KVCache
        from kempnerforge_b200.models.transformer import Transformer

        model = _build(lambda: Transformer(_config(c, n_layers=c["layers"], max_seq_len=2048)))
        model._rope_cos = model._rope_sin = None   # the tables are built in fp32 at first use
        _fill(model, g)
        s["model"] = model.eval()
        s["caches"] = [KVCache(c["batch"], c["ctx"] + 48, c["kv"], hd, BF, torch.device(DEV)) for _ in range(c["layers"])]
        for cache in s["caches"]:
            cache.k[:, : c["ctx"]].normal_(0.0, 1.0, generator=g)
            cache.v[:, : c["ctx"]].normal_(0.0, 1.0, generator=g)
        s["tokens"] = torch.randint(0, c["vocab"], (c["batch"], 1), device=DEV, generator=g)
    elif kind == "packed":
        from kempnerforge_b200.models.attention import Attention

        att = _build(lambda: Attention(c["dim"], c["heads"], c["kv"]))
        _fill(att, g)
        s["att"] = att
        s["cos"], s["sin"] = (t[: c["seq"]] for t in _rope(c))
        s["x"] = _normal(g, c["batch"], c["seq"], c["dim"]).requires_grad_(True)
        s["dy"] = _normal(g, c["batch"], c["seq"], c["dim"], std=0.01)
        s["doc"] = _doc_ids(c, seed)
    elif kind == "loss":
        s["h"] = _normal(g, c["tokens"], c["dim"]).requires_grad_(True)
        s["w"] = torch.nn.Parameter(_normal(g, c["vocab"], c["dim"], std=0.02))
        labels = torch.randint(0, c["vocab"], (c["tokens"],), device=DEV, generator=g)
        s["labels"] = torch.where(torch.rand(c["tokens"], device=DEV, generator=g) < 0.05, -100, labels)
    elif kind == "moe":
        from kempnerforge_b200.models.moe import build_moe

        layer = _build(lambda: build_moe(c["dim"], c["hidden"], c["experts"], c["topk"], router_type=c["router"],
                                         shared_experts=c["shared"], packed_experts=c["packed"]))
        _fill(layer, g)
        if c["router"] == "sigmoid_topk":
            layer.router.expert_bias.data.zero_()
            layer.router.expert_ema.fill_(1.0 / c["experts"])
        s["layer"] = layer.eval()   # eval: the sigmoid router's balancing bias stays put between passes
        s["x"] = _normal(g, c["batch"], c["seq"], c["dim"]).requires_grad_(True)
        s["dy"] = _normal(g, c["batch"], c["seq"], c["dim"], std=0.01)
    elif kind == "fp8":
        from kempnerforge_b200.models.mlp import SwiGLUMLP
        from kempnerforge_b200.ops import fp8

        mlp = _build(lambda: SwiGLUMLP(c["dim"], c["ffn"]))
        _fill(mlp, g)
        fp8.convert_model(mlp)
        s["mlp"] = mlp
        s["x"] = _normal(g, c["tokens"], c["dim"]).requires_grad_(True)
        s["dy"] = _normal(g, c["tokens"], c["dim"], std=0.01)
    elif kind == "adamw":
        from kempnerforge_b200.models.transformer import TransformerBlock
        from kempnerforge_b200.parallel.flat import FlatParamGroup
        from kempnerforge_b200.training.optimizer import FusedAdamW, build_param_groups

        block = _build(lambda: TransformerBlock(_config(c), 0))
        _fill(block, g)
        flat = FlatParamGroup("layers.0", block.named_parameters())
        opt = FusedAdamW(build_param_groups(block, 0.1), lr=3e-4, betas=(0.9, 0.95), eps=1e-8)
        opt.attach_flat_groups([flat])
        flat.grad.normal_(0.0, 1e-3, generator=g)
        flat.exp_avg.normal_(0.0, 1e-3, generator=g)
        flat.exp_avg_sq.normal_(0.0, 1e-3, generator=g).square_()
        flat.load_step(10)
        s["opt"], s["flat"], s["block"] = opt, flat, block
    else:
        raise ValueError(kind)
    return s


# --------------------------------------------------------------------------- one pass
def _grads(module):
    return {n: p.grad for n, p in module.named_parameters() if p.grad is not None}


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind in ("decode", "prefill"):
        start, n = c.get("ctx", 0), c.get("seq", 1)
        cache = s["cache"]
        cache.seq_len = start
        with torch.no_grad():
            y = s["block"](s["x"], s["cos"][start : start + n], s["sin"][start : start + n], kv_cache=cache)
        return {"y": y, "k": cache.k, "v": cache.v}
    if kind == "model":
        for cache in s["caches"]:
            cache.seq_len = c["ctx"]
        with torch.no_grad():
            logits = s["model"](s["tokens"], kv_caches=s["caches"])
        return {"logits": logits, "k": [t.k for t in s["caches"]], "v": [t.v for t in s["caches"]]}
    if kind == "train":
        x, block = s["x"], s["block"]
        x.grad = None
        if c["flat"]:
            s["flat"].zero_grad()
        else:
            block.zero_grad(set_to_none=True)
        y = block(x, s["cos"][: c["seq"]], s["sin"][: c["seq"]])
        y.backward(s["dy"])
        if c["flat"]:
            s["flat"].finalize_grads()
        return {"y": y.detach(), "dx": x.grad, "grads": _grads(block)}
    if kind == "packed":
        x, att = s["x"], s["att"]
        x.grad = None
        att.zero_grad(set_to_none=True)
        y = att(x, s["cos"], s["sin"], doc_ids=s["doc"])
        y.backward(s["dy"])
        return {"y": y.detach(), "dx": x.grad, "grads": _grads(att)}
    if kind == "loss":
        from kempnerforge_b200.ops import functional as F

        s["h"].grad = s["w"].grad = None
        loss = F.linear_cross_entropy(s["h"], s["w"], s["labels"], z_loss_weight=1e-4)
        loss.backward()
        return {"loss": loss.detach(), "dh": s["h"].grad, "dw": s["w"].grad}
    if kind == "moe":
        x, layer = s["x"], s["layer"]
        x.grad = None
        layer.zero_grad(set_to_none=True)
        y = layer(x)
        y.backward(s["dy"])
        out = {"y": y.detach(), "dx": x.grad}
        if c["packed"]:
            out["grads"] = {n: getattr(layer, n).grad for n in ("gate_w", "up_w", "down_w")}
        else:
            out["grads"] = {n: [getattr(e, n).weight.grad for e in layer.experts]
                            for n in ("gate_proj", "up_proj", "down_proj")}
        out["gate"] = layer.router.gate.weight.grad
        if layer.shared_expert is not None:
            out["shared"] = _grads(layer.shared_expert)
        return out
    if kind == "fp8":
        x, mlp = s["x"], s["mlp"]
        x.grad = None
        mlp.zero_grad(set_to_none=True)
        y = mlp(x)
        y.backward(s["dy"])
        return {"y": y.detach(), "dx": x.grad, "grads": _grads(mlp)}
    s["opt"].step()
    return {"p": s["flat"].param, "m": s["flat"].exp_avg, "v": s["flat"].exp_avg_sq}


# --------------------------------------------------------------------------- what a pass cannot do without
def _block_params(c) -> tuple[int, int]:
    """(attention, feed-forward) matrix elements of a block."""
    hd = c["dim"] // c["heads"]
    return c["dim"] * hd * (2 * c["heads"] + 2 * c["kv"]), 3 * c["dim"] * c["ffn"]


def work(case: dict) -> dict:
    c = case
    kind = c["kind"]
    hd = c["dim"] // c["heads"] if "heads" in c else 0
    if kind in ("decode", "prefill"):
        att, ff = _block_params(c)
        n, ctx = c.get("seq", 1), c.get("ctx", 0)
        t = c["batch"] * n
        kv = c["batch"] * c["kv"] * hd * 2
        pairs = n * (n + 1) / 2 + n * ctx
        return {"bytes": 2.0 * (att + ff + 2 * t * c["dim"] + kv * (ctx + n)),
                "flops": 2.0 * t * (att + ff) + 4.0 * c["batch"] * c["heads"] * hd * pairs}
    if kind == "model":
        att, ff = _block_params(c)
        kv = c["batch"] * c["kv"] * hd * 2 * (c["ctx"] + 1)
        return {"bytes": 2.0 * (c["layers"] * (att + ff + kv) + c["vocab"] * c["dim"] + c["batch"] * c["vocab"]),
                "flops": 2.0 * c["batch"] * (c["layers"] * (att + ff) + c["vocab"] * c["dim"])
                + 4.0 * c["layers"] * c["batch"] * c["heads"] * hd * (c["ctx"] + 1)}
    if kind in ("train", "packed"):
        att, ff = _block_params(c)
        w = att + (ff if kind == "train" else 0)
        t = c["batch"] * c["seq"]
        pairs = c["seq"] ** 2 / 2
        if kind == "packed":   # equal documents: what the mask leaves on average
            pairs /= (c["docs"] + 1) / 2
        # with recomputation the forward runs twice; what the result needs is one forward and one backward
        return {"bytes": 2.0 * (2 * w + 4 * t * c["dim"]),
                "flops": 6.0 * t * w + 14.0 * c["batch"] * c["heads"] * hd * pairs}
    if kind == "loss":
        n = c["tokens"] * c["dim"]
        return {"bytes": 2.0 * (2 * n + 2 * c["vocab"] * c["dim"]), "flops": 6.0 * n * c["vocab"]}
    if kind == "moe":
        t = c["batch"] * c["seq"]
        used = min(c["experts"], t * c["topk"])
        w = 3 * c["dim"] * c["hidden"]
        n_shared = 1 if c["shared"] else 0
        return {"bytes": 2.0 * ((used + c["experts"] + 2 * n_shared) * w + 4 * t * c["dim"]),
                "flops": 6.0 * t * (c["topk"] + n_shared) * w}
    if kind == "fp8":
        w = 3 * c["dim"] * c["ffn"]
        return {"bytes": 2.0 * (2 * w + 4 * c["tokens"] * c["dim"]), "flops": 6.0 * c["tokens"] * w}
    att, ff = _block_params(c)
    return {"bytes": 14.0 * (att + ff + 2 * c["dim"]), "flops": 15.0 * (att + ff)}


def tolerance(case: dict):
    kind = case["kind"]
    # bf16 results of fp32 sums: one rounding per stored tensor (2^-9 relative), a few in a row inside a layer.  Measured
    # against ``exact``: 2e-3 to 9e-3 per output of a block (1.4e-2 for a routed one); a sum in another order moves fewer bits than that.
    if kind in ("decode", "prefill", "loss"):
        return {"rel": 1e-2, "max": 0.1}
    if kind in ("train", "packed"):
        return {"rel": 1.5e-2, "max": 0.3}
    if kind == "model":
        return {"rel": 2e-2, "max": 0.15}
    if kind == "moe":
        # a token whose k-th and (k+1)-th logits are equal after rounding may go to either expert
        return {"rel": 2.5e-2, "max": 1.0 - 1e-6}
    if kind == "fp8":
        # values on the border of two fp8 numbers (3 or 2 mantissa bits) may go to either
        return {"rel": 1e-2, "max": 0.5}
    return {"rel": 4e-3, "max": 2e-2}


# --------------------------------------------------------------------------- the same in 64 bits
def _d(t):
    return t.detach().to(F64)


def _norm64(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _tables64(hd, theta, start, n):
    half = hd // 2
    inv = theta ** (-torch.arange(half, dtype=F64, device=DEV) * 2.0 / hd)
    ang = torch.outer(torch.arange(start, start + n, dtype=F64, device=DEV), inv)
    return ang.cos()[None, :, None], ang.sin()[None, :, None]


def _rope64(x, cos, sin):
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _sdpa64(q, k, v, mask):
    """q (B, Sq, H, hd), k / v (B, Sk, Hkv, hd), mask (B or 1, Sq, Sk) True = visible; one KV head at a time."""
    rep = q.shape[2] // k.shape[2]
    out = []
    for j in range(k.shape[2]):
        qj = q[:, :, j * rep : (j + 1) * rep].transpose(1, 2)
        sc = torch.matmul(qj, k[:, None, :, j].transpose(-1, -2)) / math.sqrt(q.shape[-1])
        p = torch.softmax(sc.masked_fill(~mask[:, None], float("-inf")), dim=-1)
        out.append(torch.matmul(p, v[:, None, :, j]).transpose(1, 2))
    return torch.cat(out, dim=2)


def _attn64(c, x, wq, wk, wv, wo, start=0, past=None, doc=None):
    b, n, _ = x.shape
    hd = c["dim"] // c["heads"]
    cos, sin = _tables64(hd, c["theta"], start, n)
    q = _rope64((x @ wq.t()).view(b, n, c["heads"], hd), cos, sin)
    k = _rope64((x @ wk.t()).view(b, n, c["kv"], hd), cos, sin)
    v = (x @ wv.t()).view(b, n, c["kv"], hd)
    kn, vn = k, v
    if past is not None:
        k, v = torch.cat([past[0], k], 1), torch.cat([past[1], v], 1)
    i = torch.arange(start, start + n, device=DEV)[:, None]
    mask = (torch.arange(k.shape[1], device=DEV)[None] <= i)[None]
    if doc is not None:
        mask = mask & (doc[:, :, None] == doc[:, None, :])
    return _sdpa64(q, k, v, mask).reshape(b, n, -1) @ wo.t(), kn, vn


def _block64(c, x, w, start=0, past=None):
    a, kn, vn = _attn64(c, _norm64(x, w["attention_norm.weight"]), *(w[f"attention.{t}_proj.weight"] for t in "qkvo"),
                        start=start, past=past)
    x = x + a
    n = _norm64(x, w["mlp_norm.weight"])
    h = torch.nn.functional.silu(n @ w["mlp.gate_proj.weight"].t()) * (n @ w["mlp.up_proj.weight"].t())
    return x + h @ w["mlp.down_proj.weight"].t(), kn, vn


def _weights64(module, grad=False):
    return {n: _d(p).requires_grad_(grad) for n, p in module.named_parameters()}


def _cache64(cache, ctx, kn, vn):
    k, v = _d(cache.k), _d(cache.v)
    k[:, ctx : ctx + kn.shape[1]] = kn
    v[:, ctx : ctx + vn.shape[1]] = vn
    return k, v


def _q8(t, e5m2=False):
    """Tensorwise dynamic fp8: scale to the format's range by the largest magnitude, round, scale back."""
    top, dt = (57344.0, torch.float8_e5m2) if e5m2 else (448.0, torch.float8_e4m3fn)
    f = t.to(BF).float()
    scale = top / f.abs().max()
    return (f * scale).clamp(-top, top).to(dt).to(F64) / scale.to(F64)


def _exact_fp8(s):
    x = _d(s["x"])
    wg, wu, wd = (_d(getattr(s["mlp"], n).weight) for n in ("gate_proj", "up_proj", "down_proj"))
    f = wg.shape[0]
    wgu, qx, qd = _q8(torch.cat([wg, wu])), _q8(x), _q8(wd)
    gu = (qx @ wgu.t()).to(BF).to(F64)
    g, u = gu[:, :f], gu[:, f:]
    sg = torch.sigmoid(g)
    h = (g * sg * u).to(BF).to(F64)
    qh = _q8(h)
    dy = _q8(s["dy"], True)
    dh = (dy @ qd).to(BF).to(F64)
    dgu = torch.cat([dh * u * sg * (1 + g * (1 - sg)), dh * g * sg], 1).to(BF).to(F64)
    qdgu = _q8(dgu, True)
    dwgu = qdgu.t() @ qx
    return {"y": qh @ qd.t(), "dx": qdgu @ wgu, "grads": {"gate_proj.weight": dwgu[:f], "up_proj.weight": dwgu[f:],
                                                         "down_proj.weight": dy.t() @ qh}}


def _exact_moe(s):
    c, layer = s["c"], s["layer"]
    x = _d(s["x"]).requires_grad_(True)
    xf = x.reshape(-1, c["dim"])
    gate = _d(layer.router.gate.weight).requires_grad_(True)
    logits = xf @ gate.t()
    seen = logits.detach().to(BF).to(F64)   # the router sees bf16 logits: its choice is made on those
    score = torch.sigmoid if c["router"] == "sigmoid_topk" else (lambda t: torch.softmax(t, -1))
    _, idx = torch.topk(score(seen), c["topk"], dim=-1)
    wts = score(logits).gather(1, idx)
    wts = wts / wts.sum(-1, keepdim=True)
    out = torch.zeros_like(xf)
    ws = []
    for e in range(c["experts"]):
        if c["packed"]:
            w = [_d(getattr(layer, n)[e]).t().contiguous().requires_grad_(True) for n in ("gate_w", "up_w", "down_w")]
        else:
            w = [_d(getattr(layer.experts[e], n).weight).requires_grad_(True) for n in ("gate_proj", "up_proj", "down_proj")]
        ws.append(w)
        tok, slot = (idx == e).nonzero(as_tuple=True)
        xe = xf[tok]
        y = (torch.nn.functional.silu(xe @ w[0].t()) * (xe @ w[1].t())) @ w[2].t()
        out = out.index_add(0, tok, y * wts[tok, slot, None])
    sh = {}
    if layer.shared_expert is not None:
        sh = _weights64(layer.shared_expert, True)
        out = out + (torch.nn.functional.silu(xf @ sh["gate_proj.weight"].t()) * (xf @ sh["up_proj.weight"].t())) \
            @ sh["down_proj.weight"].t()
    out.backward(_d(s["dy"]).reshape(out.shape))
    res = {"y": out.detach().view(x.shape), "dx": x.grad}
    grad = lambda t: t.grad if t.grad is not None else torch.zeros_like(t)  # noqa: E731
    per = [[grad(w[i]) for w in ws] for i in range(3)]
    if c["packed"]:
        res["grads"] = {n: torch.stack([t.t() for t in per[i]]) for i, n in enumerate(("gate_w", "up_w", "down_w"))}
    else:
        res["grads"] = {n: per[i] for i, n in enumerate(("gate_proj", "up_proj", "down_proj"))}
    res["gate"] = gate.grad
    if sh:
        res["shared"] = {n: t.grad for n, t in sh.items()}
    return res


def exact(case: dict, seed: int):
    s = prepare(case, seed)
    c, kind = s["c"], case["kind"]
    if kind in ("decode", "prefill"):
        ctx = c.get("ctx", 0)
        past = (_d(s["cache"].k[:, :ctx]), _d(s["cache"].v[:, :ctx])) if ctx else None
        y, kn, vn = _block64(c, _d(s["x"]), _weights64(s["block"]), ctx, past)
        k, v = _cache64(s["cache"], ctx, kn, vn)
        return {"y": y, "k": k, "v": v}
    if kind == "model":
        m = s["model"]
        h = _d(m.token_embedding.embedding.weight)[s["tokens"]]
        ks, vs = [], []
        for layer, cache in zip(m.layers.values(), s["caches"]):
            past = (_d(cache.k[:, : c["ctx"]]), _d(cache.v[:, : c["ctx"]]))
            h, kn, vn = _block64(c, h, _weights64(layer), c["ctx"], past)
            k, v = _cache64(cache, c["ctx"], kn, vn)
            ks.append(k)
            vs.append(v)
        logits = _norm64(h, _d(m.norm.weight)) @ _d(m.output_head.proj.weight).t()
        return {"logits": logits, "k": ks, "v": vs}
    if kind == "train":
        w = _weights64(s["block"], True)
        x = _d(s["x"]).requires_grad_(True)
        y = _block64(c, x, w)[0]
        y.backward(_d(s["dy"]))
        return {"y": y.detach(), "dx": x.grad, "grads": {n: t.grad for n, t in w.items()}}
    if kind == "packed":
        w = _weights64(s["att"], True)
        x = _d(s["x"]).requires_grad_(True)
        y = _attn64(c, x, *(w[f"{t}_proj.weight"] for t in "qkvo"), doc=s["doc"])[0]
        y.backward(_d(s["dy"]))
        return {"y": y.detach(), "dx": x.grad, "grads": {n: t.grad for n, t in w.items()}}
    if kind == "loss":
        h, w, lab = _d(s["h"]), _d(s["w"]), s["labels"]
        valid = lab != -100
        n = valid.sum().clamp_min(1)
        logits = h @ w.t()
        lse = torch.logsumexp(logits, -1)
        picked = logits.gather(1, lab.clamp_min(0)[:, None])[:, 0]
        loss = ((lse - picked) * valid).sum() / n + 1e-4 * (lse.square() * valid).sum() / n
        d = torch.exp(logits - lse[:, None]) * (1 + 2e-4 * lse)[:, None]
        d[torch.arange(lab.numel(), device=DEV), lab.clamp_min(0)] -= 1.0
        d *= (valid / n)[:, None]
        return {"loss": loss, "dh": d @ w, "dw": d.t() @ h}
    if kind == "moe":
        return _exact_moe(s)
    if kind == "fp8":
        return _exact_fp8(s)
    f = s["flat"]
    lr, b1, b2, eps, wd, step = 3e-4, 0.9, 0.95, 1e-8, 0.1, 11
    p, g, m, v = _d(f.param), _d(f.grad), _d(f.exp_avg), _d(f.exp_avg_sq)
    p[: f.n_decay] *= 1 - lr * wd
    m = b1 * m + (1 - b1) * g
    v = b2 * v + (1 - b2) * g * g
    p -= lr / (1 - b1**step) * m / (v.sqrt() / math.sqrt(1 - b2**step) + eps)
    return {"p": p, "m": m, "v": v}
