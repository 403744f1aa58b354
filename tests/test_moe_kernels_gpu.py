"""Sort, router gradient and the expert feed-forward over separate weights at the edges of their ranges."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


@pytest.mark.parametrize("slots,e", [(1, 1), (31, 8), (1024, 64), (1025, 8), (10662, 64), (5000, 256), (70000, 3)])
@pytest.mark.parametrize("skew", [False, True])
def test_stable_sort_by_expert(native_lib, slots, e, skew):
    ex = torch.randint(0, e, (slots,), device=DEV, generator=_gen(slots))
    if skew:
        ex = torch.where(torch.rand(slots, device=DEV, generator=_gen(1)) < 0.9, e - 1, ex)
    off, row, slot = native_lib.moe_sort(ex, e)
    order = torch.argsort(ex, stable=True)
    assert torch.equal(slot.long(), order)
    assert torch.equal(row.long()[order], torch.arange(slots, device=DEV))
    assert torch.equal(off.long(), torch.cat([torch.zeros(1, dtype=torch.long, device=DEV), torch.bincount(ex, minlength=e).cumsum(0)]))


@pytest.mark.parametrize("sigmoid", [False, True])
@pytest.mark.parametrize("t,e,k,dtype", [(1, 2, 1, torch.float32), (77, 8, 2, torch.bfloat16), (1777, 64, 6, torch.bfloat16),
                                         (5000, 160, 8, torch.float32), (333, 256, 8, torch.float32)])
def test_router_gradient_matches_autograd_of_the_formulas(native_lib, sigmoid, t, e, k, dtype):
    """Against the differentiable formulas (taken with create_graph) in the same fp32 arithmetic; the native scores use the
    fast exponential (2^-21 relative)."""
    from kempnerforge_b200.ops import moe_ops

    logits = torch.randn(t, e, device=DEV, generator=_gen(1)).to(dtype).requires_grad_(True)
    bias = (0.1 * torch.randn(e, device=DEV, generator=_gen(2))).to(dtype).requires_grad_(True) if sigmoid else None
    w, idx, counts, mean, z = moe_ops.route(logits, bias, sigmoid, k)
    loss = (w * torch.randn(t, k, device=DEV, generator=_gen(3))).sum() + 50 * (mean * torch.arange(e, device=DEV)).sum() + z * t
    wrt = [logits] + ([bias] if sigmoid else [])
    got = torch.autograd.grad(loss, wrt, retain_graph=True)
    want = torch.autograd.grad(loss, wrt, create_graph=True)
    for a, b in zip(got, want):
        assert a.dtype == b.dtype
        tol = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-14
        assert float((a.float() - b.float()).norm()) <= tol * float(b.float().norm())


@pytest.mark.parametrize("sigmoid", [False, True])
@pytest.mark.parametrize("t,e,k,std", [(1777, 64, 6, 1.0), (5000, 160, 8, 3.0), (2048, 8, 2, 5.0)])
@pytest.mark.parametrize("zloss", [0.0, 0.5])
def test_router_gradient_of_fp32_logits_is_as_close_to_64_bits_as_fp32_operations(native_lib, sigmoid, t, e, k, std, zloss):
    from kempnerforge_b200.ops import moe_ops

    logits = (std * torch.randn(t, e, device=DEV, generator=_gen(1))).requires_grad_(True)
    bias = 0.1 * torch.randn(e, device=DEV, generator=_gen(2)) if sigmoid else None
    w, idx, _, mean, z = moe_ops.route(logits, bias, sigmoid, k)
    dw, dm = torch.randn(t, k, device=DEV, generator=_gen(3)), torch.randn(e, device=DEV, generator=_gen(4))
    loss = (w * dw).sum() + (mean * dm).sum() + z * zloss
    got = torch.autograd.grad(loss, logits, retain_graph=True)[0]
    fp32 = torch.autograd.grad(loss, logits, create_graph=True)[0].detach()
    x = logits.detach().double().requires_grad_(True)
    s = torch.sigmoid(x + bias.double()) if sigmoid else torch.softmax(x, -1)
    sel = s.gather(1, idx)
    total = (sel / sel.sum(-1, keepdim=True) * dw.double()).sum() + (s.mean(0) * dm.double()).sum()
    want = torch.autograd.grad(total + zloss * torch.logsumexp(x, -1).square().mean(), x)[0]
    # the two differ in the order of their sums alone: 5 % of the error (the fast exponential adds 7 %)
    assert float((got.double() - want).norm()) <= 1.05 * float((fp32.double() - want).norm())


@pytest.mark.parametrize("counts", [[256], [128, 128, 128, 128], [5, 0, 300, 77, 130, 1], [0, 0, 513], [400, 17] + [3] * 30])
@pytest.mark.parametrize("extra", [0, 64])
def test_experts_with_separate_weights_match_the_packed_path(native_lib, counts, extra):
    """Same rows, same matrices: stacked into packed tensors against one tensor map per expert (bit for bit where the
    reduction is the same: everything but the input gradient's accumulation)."""
    from kempnerforge_b200.ops import grouped

    e, d, f = len(counts), 192, 320
    rows = sum(counts)
    x = torch.randn(rows + extra, d, device=DEV, generator=_gen(1)).bfloat16()
    ws = [[(torch.randn(*s, device=DEV, generator=_gen(9 * i + j)) * 0.05).bfloat16().requires_grad_(True) for i in range(e)]
          for j, s in enumerate(((f, d), (f, d), (d, f)))]
    off = grouped.offsets_of(torch.tensor(counts, device=DEV))
    dy = torch.randn(rows + extra, d, device=DEV, generator=_gen(3)).bfloat16()
    xa = x.clone().requires_grad_(True)
    ya = grouped.separate_ffn(xa, off, *ws)
    assert ya is not None
    ga = torch.autograd.grad(ya, [xa, *ws[0], *ws[1], *ws[2]], dy)
    xb = x.clone().requires_grad_(True)
    packed = [torch.stack([w.detach() for w in g]).requires_grad_(True) for g in ws]
    yb = grouped.grouped_ffn(xb, None, *packed, "nk", offsets=off)
    gb = torch.autograd.grad(yb, [xb, *packed], dy)
    assert native_lib.read_status() == 0
    assert torch.equal(ya[:rows], yb[:rows])
    assert torch.equal(ga[0][:rows], gb[0][:rows])
    for j in range(3):
        assert torch.equal(torch.stack(ga[1 + j * e : 1 + (j + 1) * e]), gb[1 + j])


def test_forms_the_separate_path_does_not_cover_return_none(native_lib):
    from kempnerforge_b200.ops import grouped

    def weights(e, f, d, dtype=torch.bfloat16):
        return [[torch.zeros(s, device=DEV, dtype=dtype) for _ in range(e)] for s in ((f, d), (f, d), (d, f))]

    off = lambda e: torch.zeros(e + 1, dtype=torch.int32, device=DEV)  # noqa: E731
    x = torch.zeros(256, 128, device=DEV, dtype=torch.bfloat16)
    assert grouped.separate_ffn(x[:255], off(2), *weights(2, 128, 128)) is None          # too few rows
    assert grouped.separate_ffn(x, off(33), *weights(33, 64, 128)) is None               # too many experts
    assert grouped.separate_ffn(x, off(2), *weights(2, 72, 128)) is None                 # F off the block
    assert grouped.separate_ffn(x, off(2), *weights(2, 128, 128, torch.float32)) is None
    g, u, dn = weights(2, 128, 128)
    assert grouped.separate_ffn(x, off(2), [torch.zeros(128, 256, device=DEV, dtype=torch.bfloat16)[:, ::2]] * 2, u, dn) is None


@pytest.mark.parametrize("counts", [[1], [32, 31, 33], [96, 97, 95, 0], [256, 257, 255], [0, 513, 0, 289, 2], [192, 193, 161, 160] * 4, [7] * 250])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("n,k", [(136, 128), (264, 192)])
def test_grouped_products_on_token_tiles(native_lib, counts, b_mn, n, k):
    """All four products against fp32 at the edges of the token tiles and with partial blocks of weight rows; rows that belong to no
    expert are not written, and what they hold (NaN) reaches no other row."""
    e, rows = len(counts), sum(counts)
    extra = 40
    off = torch.zeros(e + 1, dtype=torch.int32, device=DEV)
    off[1:] = torch.tensor(counts, device=DEV).cumsum(0)
    expert = torch.repeat_interleave(torch.arange(e, device=DEV), torch.tensor(counts, device=DEV))
    gen = _gen(rows)

    def rand(*s, std=1.0):
        return (std * torch.randn(*s, device=DEV, generator=gen)).bfloat16()

    def padded(t):
        return torch.cat([t, torch.full((extra, t.shape[1]), float("nan"), device=DEV, dtype=t.dtype)])

    shape = (e, k, n) if b_mn else (e, n, k)
    w, w2 = rand(*shape, std=0.1), rand(*shape, std=0.1)
    mats = [(v if b_mn else v.transpose(1, 2)).float() for v in (w, w2)]   # (E, K, N)
    a = rand(rows, 2 * k)
    gu = rand(rows, 2 * n)
    by = lambda x, m: torch.bmm(x.float()[:, None], m[expert])[:, 0]      # noqa: E731

    def fresh(cols):
        return torch.full((rows + extra, cols), 77.0, device=DEV, dtype=torch.bfloat16)

    def check(got, want, size, rel=2.0**-7):
        # a rounding to bf16 (2^-8 of the value) and the sum: every 16 products are added to an accumulator that keeps 23 bits of the
        # larger one, 2 k / 16 <= 24 times at most, so 2^-18 of the sum of magnitudes
        assert ((got[:rows].float() - want).abs() <= want.abs() * rel + size * 2.0**-18).all()
        assert (got[rows:] == 77.0).all()

    a1 = a[:, :k].contiguous()
    big = [by(v.abs(), m.abs()) for v, m in ((a1, mats[0]), (a1, mats[1]), (a[:, k:], mats[1]))]
    y = fresh(n)
    native_lib.grouped_experts(0, padded(a1), w, None, off, n, b_mn, y)
    want = by(a1, mats[0])
    check(y, want, big[0])
    h, pre = fresh(n), fresh(2 * n)
    native_lib.grouped_experts(1, padded(a1), w, w2, off, n, b_mn, h, pre)
    up = by(a1, mats[1])
    check(pre, torch.cat([want, up], 1), torch.cat(big[:2], 1))
    check(h, torch.nn.functional.silu(pre[:rows, :n].float()) * pre[:rows, n:].float(), 1e-2)
    d = fresh(2 * n)
    native_lib.grouped_experts(2, padded(a1), w, None, off, n, b_mn, d, padded(gu))
    g, u, dh = gu[:, :n].float(), gu[:, n:].float(), want.bfloat16().float()
    s = torch.sigmoid(g)
    check(d, torch.cat([dh * u * s * (1 + g * (1 - s)), dh * g * s], 1), 5 * torch.cat([big[0]] * 2, 1),   # |u|, |g| up to 5
          rel=2.0**-6)   # a whole step of dh (2^-7) where the two sums round apart, and the rounding of the product
    dx = fresh(n)
    native_lib.grouped_experts(3, padded(a), w, w2, off, n, b_mn, dx)
    check(dx, want + by(a[:, k:], mats[1]), big[0] + big[2])
    assert native_lib.read_status() == 0
