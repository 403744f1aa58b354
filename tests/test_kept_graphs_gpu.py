"""Backward passes over a kept graph: every pass sees the values the forward saved."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


@pytest.mark.parametrize("form", ["separate", "nk", "kn"])
@pytest.mark.parametrize("counts", [[300, 17, 0, 200], [64, 512]])
def test_experts_give_the_same_gradients_again(native_lib, form, counts):
    from kempnerforge_b200.ops import grouped

    e, d, f, rows = len(counts), 128, 192, sum(counts)
    x = torch.randn(rows, d, device=DEV, generator=_gen(1)).bfloat16().requires_grad_(True)
    shapes = ((f, d), (f, d), (d, f))
    ws = [[(torch.randn(*s, device=DEV, generator=_gen(9 * i + j)) * 0.05).bfloat16() for i in range(e)] for j, s in enumerate(shapes)]
    off = grouped.offsets_of(torch.tensor(counts, device=DEV))
    if form == "separate":
        flat = [w.requires_grad_(True) for g in ws for w in g]
        y = grouped.separate_ffn(x, off, *ws)
        node = "_SeparateFFNFn"
    else:
        flat = [torch.stack([w if form == "nk" else w.t().contiguous() for w in g]).requires_grad_(True) for g in ws]
        y = grouped.grouped_ffn(x, None, *flat, form, offsets=off)
        node = "_GroupedFFNFn"
    assert type(y.grad_fn).__name__.startswith(node)
    dy = torch.randn(rows, d, device=DEV, generator=_gen(3)).bfloat16()
    first = [t.clone() for t in torch.autograd.grad(y, [x, *flat], dy, retain_graph=True)]
    again = [t.clone() for t in torch.autograd.grad(y, [x, *flat], dy, retain_graph=True)]
    last = torch.autograd.grad(y, [x, *flat], dy)
    assert native_lib.read_status() == 0
    assert all(bool((g != 0).any()) for g in (first[0], *first[1 : 1 + (form == "separate")]))
    for a, b, c in zip(first, again, last):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("slot", [False, True])
@pytest.mark.parametrize("factor", [1.0, 0.37])
def test_loss_gives_the_same_gradients_again(native_lib, slot, factor):
    from kempnerforge_b200.ops import functional as F

    t, v, d = 300, 1000, 128
    h = torch.randn(t, d, device=DEV, generator=_gen(0)).bfloat16().requires_grad_(True)
    w = (torch.randn(v, d, device=DEV, generator=_gen(1)) * 0.05).bfloat16().requires_grad_(True)
    lab = torch.randint(0, v, (t,), device=DEV, generator=_gen(2))
    one = torch.autograd.grad(F.linear_cross_entropy(h, w, lab, 1e-3), [h, w])
    f = float(torch.tensor(factor).bfloat16())
    want = [(g.float() * f).bfloat16() for g in one]
    if slot:
        w._kf_grad = torch.zeros_like(w)

    def grads(loss, **kw):
        if not slot:
            return torch.autograd.grad(loss, [h, w], **kw)
        w._kf_grad_live = False
        return torch.autograd.grad(loss, [h], **kw)[0], w._kf_grad.clone()

    loss = F.linear_cross_entropy(h, w, lab, 1e-3) * factor
    for keep in (True, True, False):
        for a, b in zip(grads(loss, retain_graph=keep), want):
            assert torch.equal(a, b)
    assert native_lib.read_status() == 0
