"""The generation step checked in native code: the same answers as the checks in Python, and everything that is not a plain block
left to them."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _rand(*shape, seed=0, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (scale * torch.randn(*shape, device=DEV, generator=g)).bfloat16()


def _block(dim=256, heads=4, kv=2, ffn=512, batch=1, room=96, **over):
    from kempnerforge_b200.config import ModelConfig
    from kempnerforge_b200.models.attention import KVCache
    from kempnerforge_b200.models.transformer import TransformerBlock

    torch.manual_seed(1)
    cfg = ModelConfig(dim=dim, n_layers=1, n_heads=heads, n_kv_heads=kv, vocab_size=64, ffn_hidden_dim=ffn, max_seq_len=128, **over)
    block = TransformerBlock(cfg, 0).to(DEV, torch.bfloat16).eval()
    cache = KVCache(batch, room, kv, dim // heads, torch.bfloat16, torch.device(DEV))
    for i, t in enumerate((cache.k, cache.v)):
        t.copy_(_rand(*t.shape, seed=20 + i))
    cache.seq_len = 40
    x, half = _rand(batch, 1, dim, seed=2), dim // heads // 2
    ang = torch.rand(1, half, device=DEV)
    return block, cache, x, ang.cos(), ang.sin()


@pytest.mark.parametrize("dim,heads,kv,ffn,batch", [(768, 12, 12, 2048, 1), (512, 8, 2, 1024, 1), (1024, 8, 4, 768, 1), (1024, 8, 8, 1024, 5), (512, 8, 2, 1024, 3),
                                                    (768, 12, 12, 2048, 8),                                                     (512, 4, 1, 520, 33), (256, 2, 2, 512, 256)])
def test_a_step_has_the_bits_of_the_path_that_python_checks(native_lib, monkeypatch, dim, heads, kv, ffn, batch):
    block, cache, x, cos, sin = _block(dim, heads, kv, ffn, batch)
    k, v = cache.k.clone(), cache.v.clone()
    real, used = native_lib.blocks_decode, []
    monkeypatch.setattr(native_lib, "blocks_decode", lambda *a: used.append(real(*a)) or used[-1])
    with torch.no_grad():
        y = block(x, cos, sin, kv_cache=cache)
        assert used[-1] is not None and cache.seq_len == 41 and native_lib.read_status() == 0
        got = y, cache.k.clone(), cache.v.clone()
        cache.k.copy_(k), cache.v.copy_(v)
        cache.seq_len = 40
        monkeypatch.setattr(native_lib, "blocks_decode", lambda *a: None)
        want = block(x, cos, sin, kv_cache=cache), cache.k, cache.v
    assert cache.seq_len == 41 and all(torch.equal(a, b) for a, b in zip(got, want))


def _set(target, name, value):
    return lambda b, c: setattr(target(b, c), name, value)


def _none(*a):
    raise AssertionError("heads of 128 or one sequence: no other attention is asked for")


class _Sub(torch.nn.Parameter):
    pass


CHANGES = {
    "attention hook": lambda b, c: b.attention.register_forward_hook(lambda m, a, o: o),
    "mlp pre-hook": lambda b, c: b.mlp.register_forward_pre_hook(lambda m, a: None),
    "norm hook": lambda b, c: b.mlp_norm.register_forward_hook(lambda m, a, o: o),
    "replaced forward": lambda b, c: setattr(b.attention, "forward", b.attention.forward),
    "tensor parallel attention": _set(lambda b, c: b.attention, "tp", object()),
    "tensor parallel mlp": _set(lambda b, c: b.mlp, "tp", object()),
    "captured weights": _set(lambda b, c: b.attention, "capture_attention_weights", True),
    "fp8 block": _set(lambda b, c: b, "_kf_fp8_block", True),
    "fp8 flag": _set(lambda b, c: b, "fp8", True),
    "fp8 weight": _set(lambda b, c: b.mlp.down_proj.weight, "_kf_fp8", True),
    "sharded": lambda b, c: setattr(b.attention.q_proj.weight, "_kf_flat", type("Unit", (), {"sharded": True})()),
    "another norm": lambda b, c: setattr(b, "attention_norm", torch.nn.LayerNorm(256, device=DEV, dtype=torch.bfloat16)),
    "another mlp": lambda b, c: setattr(b, "mlp", torch.nn.Sequential()),
    "fp32 weight": lambda b, c: setattr(b.mlp.up_proj, "weight", torch.nn.Parameter(b.mlp.up_proj.weight.float())),
    "weight subclass": lambda b, c: setattr(b.mlp.up_proj, "weight", _Sub(b.mlp.up_proj.weight.detach())),
    "strided weight": lambda b, c: setattr(b.attention.o_proj, "weight", torch.nn.Parameter(b.attention.o_proj.weight.detach().t())),
    "weight off 16 bytes": lambda b, c: setattr(b.mlp.up_proj, "weight", torch.nn.Parameter(
        torch.zeros(512 * 256 + 1, device=DEV, dtype=torch.bfloat16)[1:].view(512, 256))),
    "another width": lambda b, c: setattr(b.mlp.up_proj, "weight", torch.nn.Parameter(b.mlp.up_proj.weight.detach()[:256])),
    "no weight": lambda b, c: setattr(b.mlp.up_proj, "weight", None),
    "cache subclass": lambda b, c: setattr(c, "__class__", type("Other", (type(c),), {})),
    "full cache": lambda b, c: setattr(c, "seq_len", 96),
    "negative position": lambda b, c: setattr(c, "seq_len", -1),
    "fp32 cache": lambda b, c: setattr(c, "v", c.v.float()),
    "other heads in the cache": lambda b, c: setattr(c, "k", c.k[:, :, :1].contiguous()),
    "strided cache": lambda b, c: setattr(c, "k", c.k.transpose(1, 2).contiguous().transpose(1, 2)),
    "cache on the host": lambda b, c: setattr(c, "v", c.v.cpu()),
}


@pytest.mark.parametrize("what", CHANGES)
def test_what_is_not_a_plain_block_is_left_to_python(native_lib, what):
    block, cache, x, cos, sin = _block()
    with torch.no_grad():
        assert native_lib.blocks_decode([block], [cache], x, cos, sin, _none) is not None
    cache.seq_len = 40
    k = cache.k.clone()
    CHANGES[what](block, cache)
    at = cache.seq_len
    with torch.no_grad():
        assert native_lib.blocks_decode([block], [cache], x, cos, sin, _none) is None
    assert cache.seq_len == at and (cache.k.shape != k.shape or torch.equal(cache.k, k))


def test_inputs_that_the_native_step_refuses(native_lib):
    block, cache, x, cos, sin = _block()
    call = lambda x=x, cos=cos, sin=sin, blocks=(block,), caches=(cache,), foreign=_none: (  # noqa: E731
        native_lib.blocks_decode(list(blocks), list(caches), x, cos, sin, foreign))
    off = lambda t: torch.empty(t.numel() + 1, device=DEV, dtype=t.dtype)[1:].view(t.shape).copy_(t)  # noqa: E731
    with torch.no_grad():
        for bad in (x.float(), x.expand(1, 2, 256).contiguous(), x[0], x[..., :128], x.repeat(2, 1, 1), off(x), x[:0], torch.nn.Parameter(x).cpu()):
            assert call(x=bad) is None
        for bad in (cos.half(), cos[:, :16].contiguous(), cos.cpu(), off(cos), cos[0], cos[:0]):
            assert call(cos=bad, sin=bad) is None
        assert call(blocks=()) is None and call(caches=()) is None and call(blocks=(block, block), caches=(cache, cache)) is None
        # the block's own hooks count when the model calls the blocks' native form in their stead
        handle = block.register_forward_hook(lambda m, a, o: o)
        assert call(foreign=None) is None and cache.seq_len == 40
        handle.remove()
        assert call(foreign=None) is not None and cache.seq_len == 41
        many = _block(512, 8, 8, 512, batch=2)   # heads of 64, several sequences: the caller's attention, if it brings one
        assert native_lib.blocks_decode([many[0]], [many[1]], *many[2:]) is None and many[1].seq_len == 40
        with pytest.raises(RuntimeError, match="dense bf16 rows"):
            native_lib.blocks_decode([many[0]], [many[1]], *many[2:], lambda q, h, hd, past: q.float())
        with pytest.raises(ZeroDivisionError):
            native_lib.blocks_decode([many[0]], [many[1]], *many[2:], lambda q, h, hd, past: 1 // 0)
        assert many[1].seq_len == 40
        with pytest.raises(TypeError):
            native_lib._steps.decode(1, 2)
    assert native_lib.read_status() == 0


@pytest.mark.parametrize("batch", [1, 3])
def test_a_cache_that_shares_its_memory_with_another_is_written_apart(native_lib, batch):
    """A lazy clone (of a beam that forks) lies in its original's memory until either is written."""
    block, cache, x, cos, sin = _block(batch=batch, heads=2)
    kept = type(cache)(batch, 96, 2, 128, torch.bfloat16, torch.device(DEV))
    kept.k, kept.v, kept.seq_len = cache.k, cache.v, cache.seq_len
    k, v = cache.k.clone(), cache.v.clone()
    cache.k, cache.v = torch._lazy_clone(kept.k), torch._lazy_clone(kept.v)
    with torch.no_grad():
        assert native_lib.blocks_decode([block], [cache], x, cos, sin, _none) is not None
    assert torch.equal(kept.k, k) and torch.equal(kept.v, v)
    rest = torch.arange(96, device=DEV) != 40
    for new, old in ((cache.k, k), (cache.v, v)):
        assert not torch.equal(new[:, 40], old[:, 40]) and torch.equal(new[:, rest], old[:, rest])
    assert cache.seq_len == 41 and native_lib.read_status() == 0


@pytest.mark.parametrize("batch,heads", [(1, 4), (3, 2), (3, 4)])
def test_a_step_without_the_module_has_the_same_bits(native_lib, monkeypatch, batch, heads):
    block, cache, x, cos, sin = _block(heads=heads, batch=batch)
    k, v = cache.k.clone(), cache.v.clone()
    with torch.no_grad():
        got = block(x, cos, sin, kv_cache=cache), cache.k.clone(), cache.v.clone()
        cache.k.copy_(k), cache.v.copy_(v)
        cache.seq_len = 40
        monkeypatch.setattr(native_lib, "_steps", False)
        want = block(x, cos, sin, kv_cache=cache), cache.k, cache.v
    assert cache.seq_len == 41 and all(torch.equal(a, b) for a, b in zip(got, want)) and native_lib.read_status() == 0
