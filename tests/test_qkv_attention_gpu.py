"""The projection + rotation + attention node and GEMMs over weights that are not adjacent, against the separate ops."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _attention(dim, heads, kv, seed=0):
    from kempnerforge_b200.models.attention import Attention

    torch.manual_seed(seed)
    with torch.device(DEV):
        return Attention(dim, heads, kv).to(torch.bfloat16)


def _run(att, x, cos, sin, ids, dy):
    att.zero_grad(set_to_none=True)
    xl = x.clone().requires_grad_(True)
    y = att(xl, cos, sin, doc_ids=ids)
    y.backward(dy)
    return [y.detach(), xl.grad] + [p.grad for p in att.parameters()]


@pytest.mark.parametrize("b,s,dim,heads,kv", [(1, 128, 256, 2, 1), (2, 333, 512, 4, 2), (1, 1000, 5120, 40, 8), (3, 700, 1024, 8, 8)])
@pytest.mark.parametrize("docs", [False, True])
def test_fused_node_matches_the_separate_ops(native_lib, monkeypatch, b, s, dim, heads, kv, docs):
    from kempnerforge_b200.models.position import precompute_rope_frequencies
    from kempnerforge_b200.ops import functional as F

    att = _attention(dim, heads, kv)
    cos, sin = precompute_rope_frequencies(128, s, 10000.0, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(1)
    x, dy = (torch.randn(b, s, dim, device=DEV, generator=g).bfloat16() for _ in range(2))
    ids = (torch.arange(s, device=DEV) // 150).expand(b, s) if docs else None
    got = _run(att, x, cos, sin, ids, dy)
    monkeypatch.setattr(F, "qkv_attention", lambda *a: None)
    want = _run(att, x, cos, sin, ids, dy)
    assert native_lib.read_status() == 0
    for a, c in zip(got, want):
        # one bf16 rounding (2^-9) fewer or more on q, k and their gradients
        assert a.shape == c.shape and float((a.float() - c.float()).norm()) <= 2.0**-6 * float(c.float().norm())


def test_calls_outside_the_fused_node_keep_their_path(native_lib):
    from kempnerforge_b200.models.position import precompute_rope_frequencies
    from kempnerforge_b200.ops import functional as F

    att = _attention(256, 2, 1)
    cos, sin = precompute_rope_frequencies(128, 200, 10000.0, device=DEV)
    x = torch.randn(1, 200, 256, device=DEV).bfloat16().requires_grad_(True)
    w = [att.q_proj.weight, att.k_proj.weight, att.v_proj.weight]
    assert F.qkv_attention(x, *w, cos, sin, None, 128) is not None
    assert F.qkv_attention(x, *w, cos.half(), sin.half(), None, 128) is None
    assert F.qkv_attention(x, *w, cos[:100], sin[:100], None, 128) is None
    assert F.qkv_attention(x[:, :100], *w, cos, sin, None, 128) is None          # fewer than one tile of rows
    assert F.qkv_attention(x, *w, cos, sin, torch.zeros(2, 200, device=DEV), 128) is None
    assert F.qkv_attention(x.float(), *w, cos, sin, None, 128) is None
    assert F.qkv_attention(x, w[0], w[1].t().contiguous().t(), w[2], cos, sin, None, 128) is None
    with torch.no_grad():
        assert F.qkv_attention(x, *w, cos, sin, None, 128) is None
    att.capture_attention_weights = True
    att(x, cos, sin)
    assert att.last_attention_weights is not None


@pytest.mark.parametrize("rows", [(4096, 1024, 1024), (2560, 2560), (3072, 64)])
def test_linear_over_weights_that_are_not_adjacent(native_lib, rows):
    from kempnerforge_b200.ops import functional as F

    g = torch.Generator(device=DEV).manual_seed(3)
    x = (torch.randn(4100, 4096, device=DEV, generator=g) * 0.5).bfloat16().requires_grad_(True)
    ws = [(torch.randn(n, 4096, device=DEV, generator=g) * 0.05).bfloat16().requires_grad_(True) for n in rows]
    y = F.fused_linear(x, ws)
    dy = torch.randn(y.shape, device=DEV, generator=g).bfloat16()
    got = torch.autograd.grad(y, [x, *ws], dy)
    w = torch.cat([t.detach() for t in ws]).double()
    assert native_lib.read_status() == 0

    def check(a, p, q):   # a bf16 rounding of an fp32 sum in any order
        want, mag = p @ q, p.abs() @ q.abs()
        assert bool(((a.double() - want).abs() <= 2.0**-8 * want.abs() + 2.0**-16 * mag).all())

    check(y, x.detach().double(), w.t())
    check(got[0], dy.double(), w)
    check(torch.cat(got[1:]), dy.double().t(), x.detach().double())


@pytest.mark.parametrize("heads", [8, 4])   # heads of 64 and of 128
def test_attention_half_of_an_expert_block_keeps_what_surrounds_it(native_lib, monkeypatch, heads):
    """Tables and hooks that the attention module serves: the same result as without the fused sub-layer."""
    from kempnerforge_b200.config import ModelConfig
    from kempnerforge_b200.models.position import precompute_rope_frequencies
    from kempnerforge_b200.models.transformer import TransformerBlock
    from kempnerforge_b200.ops import fused_block

    torch.manual_seed(0)
    cfg = ModelConfig(dim=512, n_layers=1, n_heads=heads, n_kv_heads=2, vocab_size=64, ffn_hidden_dim=256, max_seq_len=256,
                      num_experts=4, moe_top_k=2, moe_packed_experts=True)
    with torch.device(DEV):
        block = TransformerBlock(cfg, 0).to(torch.bfloat16)
    s, hd = 200, 512 // heads
    cos, sin = precompute_rope_frequencies(hd, s, 10000.0, device=DEV)
    x = torch.randn(2, s, 512, device=DEV).bfloat16()
    calls = []
    half = fused_block.attn_half
    monkeypatch.setattr(fused_block, "attn_half", lambda *a: calls.append(1) or half(*a))

    def run(c, sn):
        xl = x.clone().requires_grad_(True)
        y = block(xl, c, sn)
        (g,) = torch.autograd.grad(y.float().square().sum(), xl)
        return y.detach(), g

    want = run(cos, sin)
    assert len(calls) == 1
    packed = torch.stack([cos, sin], 1)                      # tables that are not contiguous
    apart = run(packed[:, 0], packed[:, 1])
    assert all(torch.equal(a, w) or float((a.float() - w.float()).norm()) <= 2.0**-6 * float(w.float().norm()) for a, w in zip(apart, want))
    n = len(calls)
    per_row = run(cos.expand(2, *cos.shape), sin.expand(2, *sin.shape))      # a table for every sequence: the formulas
    assert all(float((a.float() - w.float()).norm()) <= 2.0**-6 * float(w.float().norm()) for a, w in zip(per_row, want))
    seen = []
    for mod in (block.attention, block.attention_norm):
        for register in ("register_forward_pre_hook", "register_full_backward_hook"):
            handle = getattr(mod, register)(lambda *a, at=(mod, register): seen.append(at))
            run(cos, sin)
            handle.remove()
            assert seen[-1] == (mod, register)
    assert len(seen) == 4 and len(calls) == n
    run(cos, sin)
    assert len(calls) == n + 1 and native_lib.read_status() == 0
