"""Document masks evaluated per tile: the kernels that skip tiles against the fp32 reference, for ids in any order."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _ids(kind, b, s):
    g = torch.Generator(device=DEV).manual_seed(s)
    pos = torch.arange(s, device=DEV)
    if kind == "one":
        return torch.zeros(b, s, dtype=torch.long, device=DEV)
    if kind == "packed":      # documents one after the other, edges on and off the tile borders
        cuts = torch.tensor([64, 128, 129, 300, 511, 512, 700], device=DEV)
        return (pos[None, :, None] >= cuts).sum(-1).expand(b, s)
    if kind == "every":       # a document per position
        return pos.expand(b, s) * 3 - 7
    if kind == "back":        # ids that fall and return: a document in several pieces
        return ((pos // 90) % 3 - 1).expand(b, s)
    return torch.randint(-4, 5, (b, s), device=DEV, generator=g)


@pytest.mark.parametrize("kind", ["one", "packed", "every", "back", "random"])
@pytest.mark.parametrize("b,s,h,hkv,hd", [(1, 129, 2, 1, 128), (2, 1000, 4, 2, 128), (1, 640, 2, 2, 64), (1, 257, 3, 1, 128)])
@pytest.mark.parametrize("causal", [True, False])
def test_tiles_without_visible_pairs_are_skipped_without_a_trace(native_lib, kind, b, s, h, hkv, hd, causal):
    from kempnerforge_b200.ops import functional as F
    from kempnerforge_b200.ops import ref

    g = torch.Generator(device=DEV).manual_seed(1)
    q, k, v = (torch.randn(b, s, n, hd, device=DEV, generator=g).bfloat16() for n in (h, hkv, hkv))
    ids = _ids(kind, b, s)
    out, lse = native_lib.attn_fwd(q, k, v, causal, ids, 1 / math.sqrt(hd))
    want, p = ref.attention(q.float(), k.float(), v.float(), causal, ids, return_weights=True)
    # probabilities and the result rounded to bf16: 2^-8 of sum p|v| each way
    mag = torch.einsum("bhij,bjhd->bihd", p, v.float().abs().repeat_interleave(h // hkv, dim=2))
    assert native_lib.read_status() == 0
    assert bool(((out.float() - want).abs() <= 2.0**-7 * mag + 2.0**-8 * want.abs() + 1e-6).all())
    if hd != 128:
        return
    dy = torch.randn(b, s, h, hd, device=DEV, generator=g).bfloat16()
    ql, kl, vl = (t.clone().requires_grad_(True) for t in (q, k, v))
    F.attention(ql, kl, vl, causal=causal, doc_ids=ids).backward(dy)
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    ref.attention(qf, kf, vf, causal, ids).backward(dy.float())
    assert native_lib.read_status() == 0
    for a, c in ((ql, qf), (kl, kf), (vl, vf)):
        # P and dS rounded to bf16 (2^-9) inside sums of s terms: a few 2^-9 of the gradient's norm; where the exact gradient
        # is zero (a single visible key) dP - D is the difference of two fp32 sums of hd products: 2^-20 of |dout| |v| each
        assert float((a.grad.float() - c.grad).norm()) <= 2.0**-6 * float(c.grad.norm()) + 2.0**-20 * hd**0.5 * float(dy.float().norm())
