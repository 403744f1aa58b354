"""The fp8 SwiGLU feed-forward as one node: bit for bit the two fp8 Linear nodes around the SwiGLU kernel."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _mlp(dim, ffn, scale=0.05):
    from kempnerforge_b200.models.mlp import SwiGLUMLP
    from kempnerforge_b200.ops import fp8

    torch.manual_seed(0)
    with torch.device(DEV):
        mlp = SwiGLUMLP(dim, ffn).to(torch.bfloat16)
    with torch.no_grad():
        for p in mlp.parameters():
            p.normal_(0.0, scale)
    fp8.convert_model(mlp)
    return mlp


def _run(mlp, x, dy, need_x=True):
    mlp.zero_grad(set_to_none=True)
    xl = x.clone().requires_grad_(need_x)
    y = mlp(xl)
    y.backward(dy)
    return [y.detach(), xl.grad] + [p.grad for p in mlp.parameters()]


def _equal(a, b):
    return all((u is None and v is None) or torch.equal(u, v) for u, v in zip(a, b)) and len(a) == len(b)


@pytest.mark.parametrize("t,dim,ffn", [(16, 32, 16), (48, 64, 272), (400, 256, 1040), (2000, 1024, 3584)])
def test_equals_the_separate_nodes(native_lib, monkeypatch, t, dim, ffn):
    from kempnerforge_b200.ops import fp8

    mlp = _mlp(dim, ffn)
    x, dy = (torch.randn(t, dim, device=DEV).bfloat16() for _ in range(2))
    used, native = [], fp8.swiglu_mlp
    monkeypatch.setattr(fp8, "swiglu_mlp", lambda *a: used.append(native(*a)) or used[-1])
    got = _run(mlp, x, dy)
    zero = _run(mlp, torch.zeros_like(x), dy)
    for i, p in enumerate(mlp.parameters()):
        p.requires_grad_(i == 1)
    frozen = _run(mlp, x, dy, need_x=False)
    assert all(u is not None for u in used) and native_lib.read_status() == 0
    monkeypatch.setattr(fp8, "swiglu_mlp", lambda *a: None)
    assert _equal(frozen, _run(mlp, x, dy, need_x=False))
    for p in mlp.parameters():
        p.requires_grad_(True)
    assert _equal(got, _run(mlp, x, dy)) and _equal(zero, _run(mlp, torch.zeros_like(x), dy))


def test_second_backward_and_other_layers(native_lib):
    from kempnerforge_b200.ops import fp8

    mlp = _mlp(64, 128)
    x = torch.randn(3, 16, 64, device=DEV).bfloat16().requires_grad_(True)
    y = mlp(x)
    first = torch.autograd.grad(y.float().square().sum(), [x, *mlp.parameters()], retain_graph=True)
    assert _equal(first, torch.autograd.grad(y.float().square().sum(), [x, *mlp.parameters()]))
    w = [mlp.gate_proj.weight, mlp.up_proj.weight, mlp.down_proj.weight]
    assert fp8.swiglu_mlp(x[:, :5], *w) is None and fp8.swiglu_mlp(x.float(), *w) is None   # 15 rows; fp32
    assert fp8.swiglu_mlp(x, w[0], w[1], w[2].detach().clone()) is None                     # a weight that is not tagged


# Rows and hidden units at the edges of tiles: 16 is the fewest, 256 x 1024 one round of the narrowest tiles, and 2048 rows with 14 336,
# 12 288 and 10 752 units take tiles of different widths (a half of 112 or 80 columns ends inside a chunk of 32).
@pytest.mark.parametrize("t,k,f", [(16, 16, 16), (272, 144, 1024), (256, 64, 1040), (2000, 128, 14336), (2048, 256, 10752), (2544, 96, 4752), (4096, 64, 3600)])
def test_products_with_swiglu_epilogues(native_lib, t, k, f):
    """Bit for bit the product, the SwiGLU pass over what it stores and the scale of the result."""
    cu = native_lib
    torch.manual_seed(1)
    q = lambda rows, e5m2=False: cu.fp8_cast(torch.randn(rows, k, device=DEV).bfloat16(), torch.full((1,), 30.0, device=DEV), e5m2)[0]
    sa, sb = torch.full((1,), 30.0, device=DEV), torch.full((1,), 7.0, device=DEV)
    x8, w8 = q(t), q(2 * f)
    gu = cu.gemm_fp8(x8, w8, sa, sb)
    h = cu.swiglu_fwd(gu)
    *got, h_max = cu.gemm_fp8_swiglu(x8, w8, sa, sb)
    assert _equal(got, (gu, h))
    assert _equal(cu.fp8_cast(h, h_max, False, True, True), cu.fp8_cast(h, cu.fp8_scale(h), False, True, True))
    assert torch.equal(h_max.scratch[:1], cu.fp8_scale(h))
    g8, d8 = q(t, True), q(f)
    dgu = cu.swiglu_bwd(cu.gemm_fp8(g8, d8, sa, sb, a_e5m2=True), gu)
    got, dgu_max = cu.gemm_fp8_swiglu_bwd(g8, d8, sa, sb, gu)
    assert torch.equal(got, dgu)
    for maxima in (dgu_max, cu.fp8_absmax(dgu)):
        assert _equal(cu.fp8_cast(dgu, maxima, True, True, True), cu.fp8_cast(dgu, cu.fp8_scale(dgu, True), True, True, True))
        assert torch.equal(maxima.scratch[:1], cu.fp8_scale(dgu, True))
    assert native_lib.read_status() == 0


def test_saved_pre_activations_may_come_back_elsewhere(native_lib):
    """Hooks on saved tensors return copies with other strides and on other addresses."""
    mlp = _mlp(64, 272)
    x, dy = (torch.randn(48, 64, device=DEV).bfloat16() for _ in range(2))
    ref = _run(mlp, x, dy)

    def moved(t):
        if t.dim() != 2 or t.shape[0] != 48 or t.dtype != torch.bfloat16:
            return t
        return torch.empty(t.shape[0] * (t.shape[1] + 8) + 8, dtype=t.dtype, device=t.device)[8:].view(t.shape[0], -1)[:, : t.shape[1]].copy_(t)

    with torch.autograd.graph.saved_tensors_hooks(moved, lambda t: t):
        assert _equal(ref, _run(mlp, x, dy))
    with torch.autograd.graph.save_on_cpu():   # the transposed fp8 copy returns without its pitch
        assert _equal(ref, _run(mlp, x, dy))


def test_hidden_activation_is_kept_only_as_its_transposed_copy(native_lib):
    """h (48, 272) in bf16 is not among the saved tensors; without a recorded graph no transposed copy is written."""
    from kempnerforge_b200.ops import fp8

    mlp = _mlp(64, 272)
    x = torch.randn(48, 64, device=DEV).bfloat16()
    saved, wanted, quantize = [], [], fp8.quantize
    with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append((tuple(t.shape), t.dtype)) or t, lambda t: t):
        y = mlp(x)
    assert ((48, 272), torch.bfloat16) not in saved and ((272, 48), torch.uint8) in saved
    fp8.quantize = lambda *a, **k: wanted.append(k.get("want_t", False)) or quantize(*a, **k)
    try:
        with torch.no_grad():
            assert torch.equal(mlp(x), y)
    finally:
        fp8.quantize = quantize
    assert wanted and not any(wanted)


@pytest.mark.parametrize("t,dim,ffn", [(16, 32, 16), (272, 144, 1024), (2048, 256, 10752)])
def test_pre_activations_are_written_for_a_backward_only(native_lib, monkeypatch, t, dim, ffn):
    mlp = _mlp(dim, ffn)
    x = torch.randn(t, dim, device=DEV).bfloat16()
    wanted, real = [], native_lib.gemm_fp8_swiglu
    monkeypatch.setattr(native_lib, "gemm_fp8_swiglu", lambda *a, want_gu: wanted.append((want_gu, real(*a, want_gu=want_gu))) or wanted[-1][1])
    y = mlp(x)
    with torch.no_grad():
        assert torch.equal(mlp(x), y)
    for p in (mlp.gate_proj.weight, mlp.up_proj.weight):   # the gradient of the down projection alone reads the hidden activation
        p.requires_grad_(False)
    assert torch.equal(mlp(x), y)
    mlp.down_proj.weight.requires_grad_(False)
    assert torch.equal(mlp(x), y)
    assert torch.equal(mlp(x.clone().requires_grad_(True)), y)
    assert [w for w, _ in wanted] == [True, False, False, False, True]
    for w, (gu, h, maxima) in wanted:
        assert (gu is not None) == w and torch.equal(h, wanted[0][1][1])
        assert torch.equal(maxima.scratch[1 : 1 + maxima.count].max(), h.float().abs().max())
    assert native_lib.read_status() == 0


@pytest.mark.parametrize("scale", [30.0, 1e-18, 1e-19])   # ordinary, mostly infinite, all beyond fp32
@pytest.mark.parametrize("t,k,f", [(48, 64, 272), (256, 64, 1040)])
def test_values_that_are_not_finite_in_the_epilogues(native_lib, t, k, f, scale):
    """NaN operands and products beyond bf16: what the separate passes make of them, and the maxima that they find (NaN aside)."""
    cu = native_lib
    torch.manual_seed(2)
    q = lambda rows, e5m2=False: cu.fp8_cast(torch.randn(rows, k, device=DEV).bfloat16(), torch.full((1,), 30.0, device=DEV), e5m2)[0]
    sa, sb = (torch.full((1,), s, device=DEV) for s in (scale, scale))

    def same(a, b):
        return torch.equal(a.isnan(), b.isnan()) and torch.equal(a[~a.isnan()], b[~b.isnan()])

    def largest(x):
        x = x.float().abs()
        return x[~x.isnan()].max() if (~x.isnan()).any() else torch.zeros((), device=DEV)

    x8, w8, g8, d8 = q(t), q(2 * f), q(t, True), q(f)
    x8[t // 2, 3], w8[f + 5, 1], d8[7, 2] = 0x7F, 0x7F, 0x7F      # NaN of e4m3
    g8[t - 1, 0], g8[1, k - 1], g8[2, 5] = 0x7C, 0xFC, 0x7E       # inf, -inf and NaN of e5m2
    gu = cu.gemm_fp8(x8, w8, sa, sb)
    h = cu.swiglu_fwd(gu)
    for want_gu in (True, False):
        got_gu, got, maxima = cu.gemm_fp8_swiglu(x8, w8, sa, sb, want_gu)
        assert same(got, h) and (got_gu is None or same(got_gu, gu))
        assert torch.equal(maxima.scratch[1 : 1 + maxima.count].max(), largest(h))
    dh = cu.gemm_fp8(g8, d8, sa, sb, a_e5m2=True)
    for saved in (gu, torch.randn_like(gu)):
        want = cu.swiglu_bwd(dh, saved)
        got, maxima = cu.gemm_fp8_swiglu_bwd(g8, d8, sa, sb, saved)
        assert same(got, want) and torch.equal(maxima.scratch[1 : 1 + maxima.count].max(), largest(want))
    assert native_lib.read_status() == 0
