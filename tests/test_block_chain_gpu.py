"""A dense block issued by one native call per direction, against the same kernels issued op by op."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _block(dim, heads, kv, ffn, s, ac, flat):
    from kempnerforge_b200.config import ModelConfig
    from kempnerforge_b200.models.position import precompute_rope_frequencies
    from kempnerforge_b200.models.transformer import TransformerBlock
    from kempnerforge_b200.parallel.flat import FlatParamGroup

    torch.manual_seed(0)
    cfg = ModelConfig(dim=dim, n_layers=1, n_heads=heads, n_kv_heads=kv, vocab_size=64, ffn_hidden_dim=ffn, max_seq_len=max(s, 16))
    block = TransformerBlock(cfg, 0).to(DEV, torch.bfloat16)
    group = FlatParamGroup("layers.0", block.named_parameters()) if flat else None
    block.ac_mode = "full" if ac else "none"
    block.train()
    return block, group, precompute_rope_frequencies(dim // heads, s, 10000.0, device=DEV)


def _passes(block, group, tables, x, dy, n):
    if group is not None:
        group.zero_grad()
    else:
        block.zero_grad(set_to_none=True)
    out = []
    for _ in range(n):
        xl = x.clone().requires_grad_(True)
        y = block(xl, *tables)
        y.backward(dy)
        out += [y.detach(), xl.grad]
    if group is not None:
        group.finalize_grads()
    return out + [p.grad.clone() for p in block.parameters()]


# one key tile (s <= 128), or heads of 64: every sum has a fixed order and the results are equal; otherwise the dQ tiles of several
# key tiles are added in any order (fp32), which moves single bf16 roundings of dq and what follows from them
def _same(got, want, s, hd=128):
    assert len(got) == len(want)
    for a, w in zip(got, want):
        if s <= 128 or hd == 64:
            assert torch.equal(a, w)
        else:
            assert float((a.float() - w.float()).norm()) <= 2.0**-10 * float(w.float().norm())


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("ac", [False, True])
@pytest.mark.parametrize("b,s,dim,heads,kv,ffn", [(3, 100, 768, 12, 12, 2048), (4, 128, 512, 4, 4, 256), (3, 333, 768, 12, 12, 2048),
                                                  (1, 257, 2048, 16, 4, 7168), (2, 700, 1024, 8, 2, 1536)])
def test_equals_the_ops(native_lib, monkeypatch, b, s, dim, heads, kv, ffn, ac, flat):
    from kempnerforge_b200.ops import fused_block

    block, group, tables = _block(dim, heads, kv, ffn, s, ac, flat)
    g = torch.Generator(device=DEV).manual_seed(1)
    x, dy = (torch.randn(b, s, dim, device=DEV, generator=g).bfloat16() for _ in range(2))
    used = []
    native = fused_block._chain_backward
    monkeypatch.setattr(fused_block, "_chain_backward", lambda *a: used.append(native(*a)) or used[-1])
    got = _passes(block, group, tables, x, dy, 2)
    assert len(used) == 2 and all(u is not None for u in used) and native_lib.read_status() == 0
    monkeypatch.setattr(fused_block, "_chain_dims", lambda *a: None)
    _same(got, _passes(block, group, tables, x, dy, 2), s, dim // heads)
    assert len(used) == 2


def test_small_models_repeat_themselves(native_lib):
    """Heads of 64: several key tiles, and every sum has a fixed order."""
    block, _, tables = _block(768, 12, 12, 2048, 333, False, False)
    g = torch.Generator(device=DEV).manual_seed(1)
    x, dy = (torch.randn(3, 333, 768, device=DEV, generator=g).bfloat16() for _ in range(2))
    first = _passes(block, None, tables, x, dy, 1)
    for _ in range(5):
        assert all(torch.equal(a, b) for a, b in zip(first, _passes(block, None, tables, x, dy, 1)))


def test_gradient_slots_in_different_states_take_the_ops(native_lib, monkeypatch):
    from kempnerforge_b200.ops import fused_block

    block, group, tables = _block(512, 4, 4, 512, 100, False, True)
    x, dy = (torch.randn(3, 100, 512, device=DEV).bfloat16() for _ in range(2))

    def run():
        group.zero_grad()
        block.mlp.up_proj.weight._kf_grad.fill_(0.5)
        block.mlp.up_proj.weight._kf_grad_live = True
        y = block(x.clone().requires_grad_(True), *tables)
        y.backward(dy)
        group.finalize_grads()
        return [y.detach()] + [p.grad.clone() for p in block.parameters()]

    got = run()
    monkeypatch.setattr(fused_block, "_chain_dims", lambda *a: None)
    _same(got, run(), 100)


def test_second_backward_over_a_kept_graph(native_lib):
    block, _, tables = _block(512, 4, 4, 512, 100, False, False)
    x = torch.randn(3, 100, 512, device=DEV).bfloat16().requires_grad_(True)
    y = block(x, *tables)
    first = torch.autograd.grad(y.float().square().sum(), [x, *block.parameters()], retain_graph=True)
    again = torch.autograd.grad(y.float().square().sum(), [x, *block.parameters()])
    assert all(torch.equal(a, b) for a, b in zip(first, again))


def _over(block, tables, x, dy, wrap=lambda f, x: f(x)):
    """Gradients of two passes through the block in a row, their input an intermediate that nothing but the graph keeps."""
    block.zero_grad(set_to_none=True)
    xl = x.clone().requires_grad_(True)

    def body(t):
        return block(block(t * 1.5, *tables) * 0.5, *tables)

    y = wrap(body, xl)
    junk = [torch.full_like(x, float("nan")) for _ in range(8)]   # takes over memory that was given back
    y.backward(dy)
    del junk
    return [y.detach(), xl.grad] + [p.grad.clone() for p in block.parameters()]


@pytest.mark.parametrize("s", [100, 333])
def test_saved_input_comes_back_as_another_tensor(native_lib, s):
    """Saved-tensor hooks and an enclosing checkpoint hand the backward a copy, and the original is gone."""
    from torch.utils.checkpoint import checkpoint

    block, _, tables = _block(512, 4, 4, 512, s, False, False)
    g = torch.Generator(device=DEV).manual_seed(1)
    x, dy = (torch.randn(3, s, 512, device=DEV, generator=g).bfloat16() for _ in range(2))
    want = _over(block, tables, x, dy)
    assert all(bool(w.isfinite().all()) for w in want)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), lambda t: t):
        cloned = _over(block, tables, x, dy)
    with torch.autograd.graph.save_on_cpu():
        offloaded = _over(block, tables, x, dy)
    nested = _over(block, tables, x, dy, lambda f, t: checkpoint(f, t, use_reentrant=False))
    assert native_lib.read_status() == 0
    for got in (cloned, offloaded, nested):
        _same(got, want, s)


def test_weights_set_anew_between_the_passes(native_lib):
    block, _, tables = _block(512, 4, 4, 512, 100, False, False)
    x, dy = (torch.randn(3, 100, 512, device=DEV).bfloat16() for _ in range(2))

    def run(move):
        block.zero_grad(set_to_none=True)
        xl = x.clone().requires_grad_(True)
        y = block(xl, *tables)
        if move:   # the same values elsewhere; the old place is given back and overwritten
            for p in block.parameters():
                p.data = p.data.clone()
            junk = [torch.full((512 * 512,), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(16)]
        y.backward(dy)
        return [xl.grad] + [p.grad.clone() for p in block.parameters()]

    _same(run(True), run(False), 100)


def test_shapes_outside_it(native_lib, monkeypatch):
    from kempnerforge_b200.ops import fused_block

    def dims(b, s, dim, heads, kv, ffn):
        block, _, (cos, sin) = _block(dim, heads, kv, ffn, s, False, False)
        a, m = block.attention, block.mlp
        w = [block.attention_norm.weight, *(getattr(a, n + "_proj").weight for n in "qkvo"), block.mlp_norm.weight, m.gate_proj.weight,
             m.up_proj.weight, m.down_proj.weight]
        x2 = torch.zeros(b * s, dim, device=DEV, dtype=torch.bfloat16)
        return lambda cos=cos, w=w, x2=x2: fused_block._chain_dims(x2, cos, sin, w, b, s, dim, dim // heads)

    ok = dims(3, 100, 512, 4, 4, 512)
    assert ok() == (3, 100, 512, 4, 4, 128, 512)
    assert ok(cos=torch.zeros(99, 64, device=DEV)) is None
    assert dims(2, 128, 512, 4, 4, 512)() is None and dims(3, 100, 512, 4, 4, 384)() is None
    assert dims(3, 100, 512, 8, 1, 512)() is None and dims(3, 100, 768, 6, 1, 512)() is not None
    monkeypatch.setenv("KF_ATTN", "library")
    assert ok() is None
    monkeypatch.delenv("KF_ATTN")
    monkeypatch.setenv("KF_ATTN_FWD", "1")
    assert ok() is None
