"""Attention with heads of 64 and gradients: edges of the 128-key and 64-query tiles, masks, rotation, fixed order of the sums, and
which calls do not take the native kernels."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"
HD = 64


def _inputs(b, sq, sk, h, hkv, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randn(b, s, n, HD, device=DEV, generator=g).bfloat16() for s, n in ((sq, h), (sk, hkv), (sk, hkv), (sq, h))]


def _grads64(q, k, v, dout, causal, doc):
    from kempnerforge_b200.ops import ref

    q, k, v = (t.double().requires_grad_(True) for t in (q, k, v))
    out = ref.attention(q, k, v, causal=causal, doc_ids=doc)
    return torch.autograd.grad(out, (q, k, v), dout.double())


# P and dS are rounded to bf16 (2^-9 relative each, independent per element) before the products, the result once more, and D
# comes from the rounded output: below 2^-7 in the norm.
TOL = 2.0**-7


@pytest.mark.parametrize("mode", [0, 1], ids=["red", "bulk"])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("b,s,h,hkv", [(1, 1, 1, 1), (1, 63, 2, 1), (2, 65, 2, 2), (1, 128, 4, 2), (3, 333, 12, 12), (1, 1025, 8, 2)])
def test_gradients(native_lib, b, s, h, hkv, causal, mode):
    q, k, v, dout = _inputs(b, s, s, h, hkv, 11)
    prev = native_lib.attn_bwd_dq_mode(mode)
    try:
        out, lse = native_lib.attn_fwd(q, k, v, causal, None, HD**-0.5)
        got = native_lib.attn_bwd(dout, q, k, v, out, lse, causal, None, HD**-0.5)
    finally:
        native_lib.attn_bwd_dq_mode(prev)
    assert native_lib.read_status() == 0
    for a, w in zip(got, _grads64(q, k, v, dout, causal, None)):
        # one key: dq and dk are zero up to the rounding of dP - D (two sums of 64 products)
        floor = 2.0**-7 * math.sqrt(HD) if s == 1 else 0.0
        assert float((a.double() - w).norm()) <= TOL * float(w.norm()) + floor * math.sqrt(a.numel())


def test_more_keys_than_queries(native_lib):
    q, k, v, dout = _inputs(2, 100, 200, 4, 2, 5)
    out, lse = native_lib.attn_fwd(q, k, v, False, None, HD**-0.5)
    got = native_lib.attn_bwd(dout, q, k, v, out, lse, False, None, HD**-0.5)
    assert native_lib.read_status() == 0
    for a, w in zip(got, _grads64(q, k, v, dout, False, None)):
        assert float((a.double() - w).norm()) <= TOL * float(w.norm())


@pytest.mark.parametrize("s", [200, 513])
def test_documents_and_rotation_into_one_gradient(native_lib, s):
    b, h, hkv = 2, 4, 2
    q, k, v, dout = _inputs(b, s, s, h, hkv, 7)
    doc = (torch.arange(s, device=DEV) // 90).expand(b, s).contiguous()
    ang = torch.arange(s, device=DEV)[:, None] * 0.03 * torch.arange(1, HD // 2 + 1, device=DEV)[None]
    cos, sin = ang.cos().float(), ang.sin().float()
    out, lse = native_lib.attn_fwd(q, k, v, True, doc, HD**-0.5)
    dqkv = torch.empty(b, s, h + 2 * hkv, HD, device=DEV, dtype=torch.bfloat16)
    native_lib.attn_bwd(dout, q, k, v, out, lse, True, doc, HD**-0.5, dq=dqkv[:, :, :h], dk=dqkv[:, :, h : h + hkv],
                        dv=dqkv[:, :, h + hkv :], rope=(cos, sin))
    assert native_lib.read_status() == 0
    dq, dk, dv = _grads64(q, k, v, dout, True, doc)
    c, sn = cos.double()[None, :, None], sin.double()[None, :, None]
    back = lambda t: torch.cat([t[..., :32] * c + t[..., 32:] * sn, t[..., 32:] * c - t[..., :32] * sn], -1)  # noqa: E731
    want = torch.cat([back(dq), back(dk), dv], 2)
    assert float((dqkv.double() - want).norm()) <= TOL * float(want.norm())


def test_what_stays_on_the_library(native_lib):
    q, k, v, _ = _inputs(1, 128, 128, 2, 2, 3)
    assert native_lib.attn_supported(q, k, v, True, needs_grad=True)
    assert native_lib.attn_bwd_chosen(64, 8, 2896, 2896, True, False) and not native_lib.attn_bwd_chosen(64, 8, 2897, 2897, True, False)
    assert not native_lib.attn_bwd_chosen(64, 1, 128, 128, True, True) and native_lib.attn_bwd_chosen(128, 99, 4096, 4096, True, False)
    assert not native_lib.attn_supported(q, k, v, True, needs_grad=True, docs=True) and native_lib.attn_supported(q, k, v, True, docs=True)
    assert not native_lib.attn_bwd_chosen(96, 1, 64, 64, True, True)
    torch.use_deterministic_algorithms(True)
    try:
        assert not native_lib.attn_supported(q, k, v, True, needs_grad=True)
        assert not native_lib.attn_supported(q, k, v, True, needs_grad=True, docs=True) and native_lib.attn_supported(q, k, v, True)
    finally:
        torch.use_deterministic_algorithms(False)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("b,s,h,hkv", [(3, 333, 12, 12), (2, 1025, 8, 2), (1, 2048, 12, 12)])
def test_equal_inputs_give_equal_bits(native_lib, b, s, h, hkv, causal):
    q, k, v, dout = _inputs(b, s, s, h, hkv, 2)
    out, lse = native_lib.attn_fwd(q, k, v, causal, None, HD**-0.5)
    first = native_lib.attn_bwd(dout, q, k, v, out, lse, causal, None, HD**-0.5)
    for _ in range(10):
        again = native_lib.attn_bwd(dout, q, k, v, out, lse, causal, None, HD**-0.5)
        assert all(torch.equal(x, y) for x, y in zip(first, again))
    assert native_lib.read_status() == 0


def test_parts_of_the_longest_call_fit(native_lib):
    n = native_lib.attn_bwd_dq_floats
    assert n(3, 333, 333, 12, 128) == 3 * 333 * 12 * 128
    assert n(3, 333, 333, 12, 64) == 3 * 3 * 12 * 384 * 64
    for causal, s in ((True, 2896), (False, 2048)):
        assert s * s * 8 // (1 + causal) <= native_lib.HEAD64_MAX_SCORES < (s + 1) ** 2 * 8 // (1 + causal)
        assert n(1, s, s, 8, 64) <= native_lib.HEAD64_MAX_PARTS
    # sequences much shorter than a tile: the tiles, not the scores, are what a call costs
    assert native_lib.attn_bwd_chosen(64, 12 * 768, 8, 8, True, False) and not native_lib.attn_bwd_chosen(64, 12 * 769, 8, 8, True, False)


def test_documents_with_gradients_stay_in_fp32(native_lib):
    """Nothing but the result is rounded to bf16: 2^-9 relative per value."""
    from kempnerforge_b200.models.attention import Attention
    from kempnerforge_b200.ops import functional as F
    from kempnerforge_b200.ops import ref

    b, s, h, hkv = 2, 300, 4, 2
    q, k, v, dout = _inputs(b, s, s, h, hkv, 7)
    doc = (torch.arange(s, device=DEV) // 90).expand(b, s).contiguous()
    ql, kl, vl = (t.clone().requires_grad_(True) for t in (q, k, v))
    out = F.attention(ql, kl, vl, doc_ids=doc)
    got = torch.autograd.grad(out, (ql, kl, vl), dout)
    want64 = ref.attention(q.double(), k.double(), v.double(), doc_ids=doc)
    for a, w in zip((out.detach(), *got), (want64, *_grads64(q, k, v, dout, True, doc))):
        assert float((a.double() - w).norm()) <= 2.0**-9 * float(w.norm())
    # the layer takes the same way
    torch.manual_seed(0)
    att = Attention(h * HD, h, hkv).to(DEV, torch.bfloat16)
    x = torch.randn(b, s, h * HD, device=DEV).bfloat16().requires_grad_(True)
    tables = [t.cos() if i == 0 else t.sin() for i, t in enumerate([torch.rand(s, HD // 2, device=DEV) * 6] * 2)]
    w = [att.q_proj.weight, att.k_proj.weight, att.v_proj.weight]
    assert F.qkv_attention(x, *w, *tables, doc, HD) is None and F.qkv_attention(x, *w, *tables, None, HD) is not None


def test_called_by_itself_it_transforms(native_lib):
    from kempnerforge_b200.ops import functional as F

    q, k, v, dout = _inputs(2, 150, 150, 2, 2, 9)

    def loss(q, k, v, d):
        return (F.attention(q, k, v) * d).float().sum()

    got = torch.func.grad(loss, argnums=(0, 1, 2))(q, k, v, dout)
    ql, kl, vl = (t.clone().requires_grad_(True) for t in (q, k, v))
    want = torch.autograd.grad(loss(ql, kl, vl, dout), (ql, kl, vl))
    assert all(torch.equal(a, w) for a, w in zip(got, want))
    with torch.nn.attention.sdpa_kernel(torch.nn.attention.SDPBackend.MATH):   # the program's choice of kernel holds
        (first,) = torch.autograd.grad(loss(ql, kl, vl, dout), ql, create_graph=True)
        assert first.requires_grad
