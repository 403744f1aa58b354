"""Document ids in the shapes that callers hand over: one row per sequence, flat, one row for all sequences."""

import math

import pytest
import torch

DEV = "cuda"


def test_ids_are_brought_to_one_row_per_sequence_or_refused(monkeypatch):
    from kempnerforge_b200.ops import cuda as kc

    seen = []

    class _Library:
        def kf_doc_blocks(self, ids, wide, out, rng, b, s, stream):
            seen.append((b, s))
            return 0

    monkeypatch.setattr(kc, "lib", lambda: _Library())
    monkeypatch.setattr(kc, "_stream", lambda: 0)
    k = torch.zeros(2, 70, 1, 64)
    for ids in (torch.zeros(2, 70, dtype=torch.long), torch.zeros(140, dtype=torch.int32), torch.zeros(1, 70), torch.zeros(70)):
        out, rng = kc.doc_blocks(ids, k)
        assert out.shape == (2, 70) and rng.shape == (2, 2, 2)
    assert seen == [(2, 70)] * 4
    for ids in (torch.zeros(2, 69), torch.zeros(1, 140, 1, 2), torch.zeros(3, 70), torch.zeros(2, 70, device="meta")):
        with pytest.raises((RuntimeError, AssertionError)):
            kc.doc_blocks(ids, k)
    assert len(seen) == 4


@pytest.mark.gpu
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("b,shape", [(1, (300,)), (1, (1, 300)), (2, (1, 300)), (2, (600,))])
def test_attention_takes_every_shape(native_lib, grad, b, shape):
    from kempnerforge_b200.ops import functional as F
    from kempnerforge_b200.ops import ref

    g = torch.Generator(device=DEV).manual_seed(0)
    q, k, v, dy = (torch.randn(b, 300, n, 128, device=DEV, generator=g).bfloat16() for n in (4, 2, 2, 4))
    ids = (torch.arange(300, device=DEV) // 77).expand(b, 300)
    given = ids.reshape(-1)[: math.prod(shape)].view(shape)
    ql, kl, vl = (t.clone().requires_grad_(grad) for t in (q, k, v))
    out = F.attention(ql, kl, vl, causal=True, doc_ids=given)
    want = ref.attention(q.float(), k.float(), v.float(), True, ids)
    assert float((out.detach().float() - want).norm()) <= 2.0**-7 * float(want.norm())   # P and the result rounded to bf16
    if grad:
        got = torch.autograd.grad(out, [ql, kl, vl], dy)
        qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
        for a, c in zip(got, torch.autograd.grad(ref.attention(qf, kf, vf, True, ids), [qf, kf, vf], dy.float())):
            assert float((a.float() - c).norm()) <= 2.0**-6 * float(c.norm())                # dS rounded as well
    assert native_lib.read_status() == 0
