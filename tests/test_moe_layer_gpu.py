"""What a mixture-of-experts layer takes from one launch: the router's weights, losses and counts, the combination with a shared
expert, and the SwiGLU MLP as one node, each against the separate operations it stands for."""

import pytest
import torch
import torch.utils.checkpoint

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(*shape, seed, std=1.0, dtype=torch.bfloat16):
    return (std * torch.randn(*shape, device=DEV, generator=_gen(seed))).to(dtype)


@pytest.mark.parametrize("sigmoid", [False, True])
@pytest.mark.parametrize("t,e,k", [(1, 1, 1), (7, 33, 8), (1777, 64, 6), (9600, 256, 2)])
@pytest.mark.parametrize("bias_dtype", [torch.float32, torch.bfloat16])
def test_router_of_a_layer_matches_the_separate_operations(native_lib, sigmoid, t, e, k, bias_dtype):
    from kempnerforge_b200.ops import moe_ops

    logits = _randn(t, e, seed=1).requires_grad_(True)
    bias = _randn(e, seed=2, std=0.1, dtype=bias_dtype).requires_grad_(True) if sigmoid else None
    w, idx, counts, mean, z, balance = moe_ops.route_layer(logits, bias, sigmoid, k, torch.bfloat16)
    w32, idx32, counts32, mean32, z32 = moe_ops.route(logits, bias, sigmoid, k)
    assert torch.equal(idx, idx32) and torch.equal(counts, counts32) and torch.equal(w, w32.to(torch.bfloat16))
    assert torch.equal(counts, torch.bincount(idx.reshape(-1), minlength=e).float())
    # fp32 sums of t scores per expert in an order that is not fixed
    lf = logits.detach().double()
    scores = torch.sigmoid(lf + bias.detach().double()) if sigmoid else torch.softmax(lf, -1)
    assert torch.allclose(mean.double(), scores.mean(0), rtol=2e-5, atol=1e-9)
    assert torch.allclose(z.double(), torch.logsumexp(lf, -1).square().mean(), rtol=2e-5, atol=1e-12)
    want = 0.0 if sigmoid else float(e * (counts.double() / (t * k) * scores.mean(0)).sum())
    assert float(balance.detach()) == pytest.approx(want, rel=2e-5)
    assert balance.requires_grad == (not sigmoid)
    counts.zero_()   # a program that resets or reduces the counts in place changes no gradient

    # gradients: the layer's outputs against the same loss over route() and tensor operations
    dw = _randn(t, k, seed=3)
    wrt = [logits] + ([bias] if sigmoid else [])
    loss = (w * dw).sum().float() + z * 0.3 + (0 if sigmoid else balance * 5)
    frac = counts32 / (t * k)
    loss32 = (w32.to(torch.bfloat16) * dw).sum().float() + z32 * 0.3 + (0 if sigmoid else e * (frac * mean32).sum() * 5)
    got = torch.autograd.grad(loss, wrt, retain_graph=True)
    ref = torch.autograd.grad(loss32, wrt)
    diff = torch.autograd.grad(loss, wrt, create_graph=True)
    for a, b, c in zip(got, ref, diff):
        assert a.dtype == b.dtype == c.dtype
        # bf16 gradients of the same fp32 values: one rounding apart at most
        scale = float(b.float().norm()) + 1e-12
        assert float((a.float() - b.float()).norm()) <= 2.0**-9 * scale
        assert float((a.float() - c.detach().float()).norm()) <= 2.0**-7 * scale
    assert native_lib.read_status() == 0


def test_router_outputs_that_nothing_uses_ask_for_no_gradient(native_lib):
    from kempnerforge_b200.ops import moe_ops

    logits = _randn(300, 16, seed=1).requires_grad_(True)
    for pick in range(4):   # weights, mean scores, z-loss, balancing loss alone
        w, idx, counts, mean, z, balance = moe_ops.route_layer(logits, None, False, 2, torch.bfloat16)
        v = torch.arange(16, device=DEV, dtype=torch.float32)
        loss = (w.float()[:, 0].sum(), (mean * v).sum(), z, balance)[pick]
        got, = torch.autograd.grad(loss, logits, retain_graph=True)
        x = logits.detach().double().requires_grad_(True)
        p = torch.softmax(x, -1)
        top = p.gather(1, idx)   # equal logits: whichever of them was chosen
        want64 = ((top / top.sum(-1, keepdim=True))[:, 0].sum(), (p.mean(0) * v.double()).sum(),
                  torch.logsumexp(x, -1).square().mean(), 16 * (counts.double() / 600 * p.mean(0)).sum())[pick]
        want, = torch.autograd.grad(want64, x)
        assert float((got.double() - want).norm()) <= 2.0**-8 * float(want.norm())   # the gradient is rounded to bf16


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("t,k,cols", [(1, 1, 8), (777, 6, 2048), (100, 8, 264)])
def test_combination_with_a_shared_expert_has_the_bits_of_an_addition(native_lib, dtype, t, k, cols):
    from kempnerforge_b200.ops import moe_ops

    idx = torch.randint(0, 5, (t, k), device=DEV, generator=_gen(1))
    _, row, slot = moe_ops.sort_by_expert(idx, 5)
    y, w, plus, dout = _randn(t * k, cols, seed=2), _randn(t, k, seed=3, dtype=dtype), _randn(t, cols, seed=4), _randn(t, cols, seed=5)
    leaves = [v.clone().requires_grad_(True) for v in (y, w, plus)]
    out = moe_ops.combine_rows(leaves[0], leaves[1], row, slot, leaves[2])
    got = torch.autograd.grad(out, leaves, dout)
    ref = [v.clone().requires_grad_(True) for v in (y, w, plus)]
    two = moe_ops.combine_rows(ref[0], ref[1].float(), row, slot) + ref[2]
    want = torch.autograd.grad(two, ref, dout)
    assert torch.equal(out, two)
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and torch.equal(a, b)
    strided = torch.empty(t, cols + 8, device=DEV, dtype=torch.bfloat16)[:, :cols].copy_(plus)   # added by itself
    assert torch.equal(moe_ops.combine_rows(y, w, row, slot, strided), two)


@pytest.mark.parametrize("rows,d,f", [(256, 64, 128), (1777, 2048, 1408), (300, 192, 384), (2048, 256, 7296)])
def test_swiglu_mlp_as_one_node_has_the_bits_of_its_parts(native_lib, rows, d, f, monkeypatch):
    from kempnerforge_b200.models.mlp import SwiGLUMLP
    from kempnerforge_b200.ops import functional as F

    with torch.device(DEV):
        mlp = SwiGLUMLP(d, f).to(torch.bfloat16)
    x, dy = _randn(3, rows // 3, d, seed=1) if rows % 3 == 0 else _randn(rows, d, seed=1), None
    dy = _randn(*x.shape, seed=2)
    calls = []
    real = F.swiglu_mlp
    monkeypatch.setattr(F, "swiglu_mlp", lambda *a: calls.append(real(*a)) or calls[-1])

    def run(x, keep=False):
        x = x.clone().requires_grad_(True)
        y = mlp(x)
        wrt = [x, *mlp.parameters()]
        if keep:   # a graph that is kept gives the same gradients twice
            first = torch.autograd.grad(y, wrt, dy, retain_graph=True)
            again = torch.autograd.grad(y, wrt, dy)
            assert all(torch.equal(a, b) for a, b in zip(first, again))
        return y.detach(), torch.autograd.grad(mlp(x), wrt, dy)

    y1, g1 = run(x, keep=True)
    assert calls and calls[0] is not None
    with torch.no_grad():
        assert torch.equal(mlp(x), y1)
    monkeypatch.setattr(F, "swiglu_mlp", lambda *a: None)
    y2, g2 = run(x)
    assert torch.equal(y1, y2)
    for a, b in zip(g1, g2):
        assert torch.equal(a, b)
    # frozen parts
    monkeypatch.setattr(F, "swiglu_mlp", real)
    for frozen in ([mlp.down_proj], [mlp.gate_proj, mlp.up_proj], [mlp.gate_proj]):
        for m in frozen:
            m.weight.requires_grad_(False)
        xg = x.clone().requires_grad_(True)
        live = [xg, *(p for p in mlp.parameters() if p.requires_grad)]
        got = torch.autograd.grad(mlp(xg), live, dy)
        names = dict(zip(["x", *(n for n, _ in mlp.named_parameters())], g1))
        want = [names["x"], *(names[n] for n, p in mlp.named_parameters() if p.requires_grad)]
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        for m in frozen:
            m.weight.requires_grad_(True)
    assert native_lib.read_status() == 0


def test_forms_the_one_node_mlp_leaves_to_its_parts(native_lib):
    from kempnerforge_b200.ops import functional as F

    def call(rows=256, d=64, f=256, dtype=torch.bfloat16, change=None):
        x = torch.zeros(rows, d, device=DEV, dtype=dtype)
        ws = [torch.zeros(s, device=DEV, dtype=dtype) for s in ((f, d), (f, d), (d, f))]
        if change:
            ws = change(ws)
        return F.swiglu_mlp(x, *ws)

    assert call() is not None
    assert call(rows=255) is None
    assert call(d=72) is None
    assert call(f=192) is None
    assert call(dtype=torch.float32) is None
    assert call(rows=0) is None
    assert call(change=lambda w: [w[0].t().contiguous().t(), *w[1:]]) is None          # another stride
    assert call(change=lambda w: [w[0], w[1][:128].contiguous(), w[2]]) is None                     # another width
    off = torch.zeros(256 * 64 + 1, device=DEV, dtype=torch.bfloat16)[1:].view(256, 64)
    assert call(change=lambda w: [off, *w[1:]]) is None                                # off 16 bytes


def test_pre_activations_are_written_for_a_backward_only(native_lib, monkeypatch):
    """Parameters ask for gradients under no_grad too: evaluation, generation, the first pass of a checkpointed layer."""
    from kempnerforge_b200.models.mlp import SwiGLUMLP

    with torch.device(DEV):
        mlp = SwiGLUMLP(256, 384).to(torch.bfloat16)
    x = _randn(300, 256, seed=1)
    wanted, real = [], native_lib.gemm_swiglu_pair
    monkeypatch.setattr(native_lib, "gemm_swiglu_pair", lambda *a, want_gu: wanted.append(want_gu) or real(*a, want_gu=want_gu))
    y = mlp(x)
    with torch.no_grad():
        assert torch.equal(mlp(x), y)
    with torch.inference_mode():
        assert torch.equal(mlp(x), y)
    xg = x.clone().requires_grad_(True)
    again = torch.utils.checkpoint.checkpoint(mlp, xg, use_reentrant=True)
    again.sum().backward()
    for p in mlp.parameters():
        p.requires_grad_(False)
    assert torch.equal(mlp(x), y) and torch.equal(again, y)
    assert wanted == [True, False, False, False, True, False] and native_lib.read_status() == 0


@pytest.mark.parametrize("sigmoid", [False, True])
@pytest.mark.parametrize("t,e,k", [(1, 1, 1), (9, 8, 2), (300, 64, 6), (40, 256, 8), (33, 8, 8)])
def test_router_of_tokens_that_are_not_finite(native_lib, sigmoid, t, e, k):
    """A NaN is the largest, as for torch.topk: k different experts are found for every token, and its weights say what happened."""
    from kempnerforge_b200.ops import moe_ops

    clean = _randn(t, e, seed=1, dtype=torch.float32)
    logits = clean.clone()
    bad = {0: slice(0, e), t // 2: slice(e // 2, e), t - 1: slice(e - 1, e)}
    for row, cols in bad.items():
        logits[row, cols] = float("nan")
    if t > 8:
        logits[1], logits[2] = -torch.inf, torch.inf   # no score at all; every one the largest
        bad |= {1: slice(0, e), 2: slice(0, e)}
    w, idx, counts, mean, z, balance = moe_ops.route_layer(logits, None, sigmoid, k, torch.float32)
    scores = torch.sigmoid(logits) if sigmoid else torch.softmax(logits, -1)
    order = torch.where(scores.isnan(), torch.inf, scores).sort(dim=-1, descending=True, stable=True).indices[:, :k]
    rows = sorted(bad)
    assert torch.equal(idx[rows], order[rows])
    assert torch.equal(counts, torch.bincount(idx.reshape(-1), minlength=e).float()) and int(counts.sum()) == t * k
    assert torch.equal(w.isnan().any(1), scores.gather(1, idx).isnan().any(1) | (scores.gather(1, idx).sum(1) == 0))
    assert torch.equal(mean.isnan(), scores.isnan().any(0)) and not z.isfinite() and (sigmoid or balance.isnan())
    fine = [i for i in range(t) if i not in bad]
    if fine:
        w2, idx2, *_ = moe_ops.route_layer(clean, None, sigmoid, k, torch.float32)
        assert torch.equal(w[fine], w2[fine]) and torch.equal(idx[fine], idx2[fine])
    assert native_lib.read_status() == 0


@pytest.mark.parametrize("packed,router", [(True, "sigmoid_topk"), (False, "softmax_topk")])
def test_a_token_that_is_not_finite_keeps_to_itself(native_lib, packed, router):
    from kempnerforge_b200.models.moe import build_moe

    torch.manual_seed(4)
    with torch.device(DEV):
        moe = build_moe(dim=128, hidden_dim=256, num_experts=8, top_k=2, router_type=router, packed_experts=packed).to(torch.bfloat16).eval()
    x = _randn(1, 400, 128, seed=5)
    with torch.no_grad():
        want = moe(x)
        x[0, 77] = float("nan")
        got = moe(x)
    others = torch.arange(400, device=DEV) != 77
    assert got[0, 77].isnan().all() and torch.equal(got[0, others], want[0, others]) and native_lib.read_status() == 0
