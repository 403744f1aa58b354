"""Kernels and dispatch of the gradient-free block (generation, evaluation) at the edges of their tiles, against fp32."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _rand(*shape, scale=1.0, seed=None):
    g = torch.Generator(device=DEV).manual_seed(seed) if seed is not None else None
    return (torch.randn(*shape, device=DEV, generator=g) * scale).to(torch.bfloat16)


def _check_dot(got, a, b, extra=None):
    """One bf16 rounding (half an ulp: up to 2^-8 relative) of an fp32 dot product summed in any order (K 2^-24 sum|ab| bounds the
    order's effect; 2^-16 covers K up to 256 partial sums per accumulator step and the split)."""
    want = a.double() @ b.double().t()
    mag = a.double().abs() @ b.double().abs().t()
    if extra is not None:
        want, mag = want + extra.double(), mag + extra.double().abs()
    err = (got.double() - want).abs()
    assert bool((err <= 2.0**-8 * want.abs() + 2.0**-16 * mag).all()), float((err / (mag + 1e-30)).max())


@pytest.mark.parametrize("m,rows,k", [
    (1, [8], 8), (1, [4096], 4096), (3, [136], 72), (16, [128, 128, 128], 512), (17, [264, 40, 8], 520), (32, [1024], 264),
    (33, [120], 2048), (64, [256, 64], 64), (65, [392], 1000), (128, [512], 768), (129, [136, 128], 320), (256, [264], 4096),
])
def test_few_row_gemm_over_separate_weights(native_lib, monkeypatch, m, rows, k):
    monkeypatch.setattr(native_lib, "_few_rows", lambda m, n: True)
    x = _rand(m, k, scale=0.5, seed=1)
    ws = [_rand(n, k, scale=0.5, seed=2 + i) for i, n in enumerate(rows)]
    n = sum(rows)
    res = _rand(m, n, seed=9)
    buf = torch.full((m + 1, n + 8), 7.0, dtype=torch.bfloat16, device=DEV)   # a frame that must stay untouched
    out = native_lib.gemm_rows(x, ws, out=buf[:m, :n])
    plain = native_lib.gemm_rows(x, ws, residual=res)
    assert native_lib.read_status() == 0
    w = torch.cat(ws)
    _check_dot(out, x, w)
    _check_dot(plain, x, w, res)
    assert bool((buf[m:] == 7).all()) and bool((buf[:, n:] == 7).all())
    assert torch.equal(out, native_lib.gemm_rows(x, ws))                       # fixed reduction order


@pytest.mark.parametrize("m,f,k", [(1, 64, 128), (5, 72, 520), (16, 14336, 4096), (40, 200, 2048), (256, 1024, 768)])
def test_few_row_swiglu_epilogue(native_lib, m, f, k):
    x, wg, wu = _rand(m, k, seed=1), _rand(f, k, scale=k**-0.5, seed=2), _rand(f, k, scale=k**-0.5, seed=3)
    got = native_lib.swiglu_rows(x, wg, wu).double()
    g, u = x.double() @ wg.double().t(), x.double() @ wu.double().t()
    want = torch.nn.functional.silu(g) * u
    assert native_lib.read_status() == 0
    # gate and up are fp32 sums in some order (2^-16 of sum|ab|, as in _check_dot) rounded to bf16 (2^-8 relative); the
    # product has slope 1.1 |u| in the gate and |silu(g)| in up, and is rounded once more
    dg = 2.0**-8 * g.abs() + 2.0**-16 * (x.double().abs() @ wg.double().abs().t())
    du = 2.0**-8 * u.abs() + 2.0**-16 * (x.double().abs() @ wu.double().abs().t())
    bound = 1.1 * (u.abs() + du) * dg + torch.nn.functional.silu(g).abs() * du + 2.0**-8 * want.abs()
    assert bool(((got - want).abs() <= bound).all())


@pytest.mark.parametrize("m,f,k", [(2, 64, 128), (2, 72, 520), (16, 256, 768), (3, 14336, 1024)])   # small weights, tiles, a large weight
def test_operands_off_16_bytes_are_refused(native_lib, m, f, k):
    """The copies into shared memory need 16-byte steps whichever kernel takes the product: an error from the host, no launch."""
    def off(*shape):   # contiguous, two bytes further
        return torch.zeros(math.prod(shape) + 1, dtype=torch.bfloat16, device=DEV)[1:].view(shape)

    L, kc = native_lib.lib(), native_lib
    x, wg, wu, gain = _rand(m, k), _rand(f, k), _rand(f, k), _rand(k)
    h = torch.full((m, f), 7.0, dtype=torch.bfloat16, device=DEV)
    for bad in range(3):
        ops = [off(*t.shape) if i == bad else t for i, t in enumerate((x, wg, wu))]
        with pytest.raises(native_lib.NativeKernelError):
            native_lib.swiglu_rows(*ops)
    if m <= L.kf_skinny_norm_rows():
        for src, g in ((x, off(k)), (off(m, k), gain)):
            assert L.kf_gemm_skinny_norm_swiglu_bf16(src.data_ptr(), g.data_ptr(), 1e-5, wg.data_ptr(), wu.data_ptr(), h.data_ptr(), m, f, k,
                                                     k, k, k, f, 0, kc.sm_count(), kc._stream()) != 0
    torch.cuda.synchronize()
    assert native_lib.read_status() == 0 and bool((h == 7).all())


def _cache(b, room, hkv, hd, seed):
    """A cache of bounded values followed by NaNs: nothing past the visible positions may be read."""
    return _rand(b, room, hkv, hd, seed=seed), _rand(b, room, hkv, hd, seed=seed + 1)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("b,sk,h,hkv", [(1, 1, 4, 4), (2, 63, 8, 2), (1, 64, 5, 1), (3, 65, 8, 2), (1, 1000, 32, 8),
                                        (16, 129, 40, 8), (2, 4001, 4, 1), (1, 300, 16, 1), (1, 200, 20, 1), (1, 513, 34, 2)])
def test_decode_attention_over_a_strided_cache(native_lib, b, sk, h, hkv, hd):
    room = sk + 7
    k, v = _cache(b, room, hkv, hd, 3)
    k[:, sk:], v[:, sk:] = float("nan"), float("nan")
    q = _rand(b, h * hd, seed=5)
    out = torch.full((b, h * hd), 3.0, dtype=torch.bfloat16, device=DEV)
    scale = 1.0 / math.sqrt(hd)
    native_lib._check(native_lib.lib().kf_attn_decode_bf16(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), b, sk, h, hkv, hd, h * hd, h * hd, hkv * hd, k.stride(0),
        v.stride(0), scale, 0, 0, native_lib.sm_count(), torch.cuda.current_stream().cuda_stream), "decode")
    rep = h // hkv
    kd, vd = (t[:, :sk].double().repeat_interleave(rep, dim=2) for t in (k, v))
    p = torch.softmax(torch.einsum("bhd,bshd->bhs", q.double().view(b, h, hd), kd) * scale, dim=-1)
    want = torch.einsum("bhs,bshd->bhd", p, vd)
    mag = torch.einsum("bhs,bshd->bhd", p, vd.abs())
    # probabilities rounded to bf16 (2^-9 each, not all the same way) and one rounding of the result
    assert bool(((out.double().view(b, h, hd) - want).abs() <= 2.0**-8 * mag + 2.0**-8 * want.abs()).all())


def _block(kind, hd=128, heads=4, kv=2, seed=0):
    from kempnerforge_b200.config import ModelConfig
    from kempnerforge_b200.models.transformer import TransformerBlock

    extra = {"swiglu": {}, "gelu": dict(activation="gelu"), "moe": dict(num_experts=4, moe_top_k=2, moe_frequency=1)}[kind]
    cfg = ModelConfig(dim=hd * heads, n_layers=1, n_heads=heads, n_kv_heads=kv, vocab_size=256, ffn_hidden_dim=640,
                      max_seq_len=1024, **extra)
    torch.manual_seed(seed)
    with torch.device(DEV):
        block = TransformerBlock(cfg, 0).to(torch.bfloat16)
    return block.eval(), cfg


def _tables(hd, n=1024):
    from kempnerforge_b200.models.position import precompute_rope_frequencies

    return precompute_rope_frequencies(hd, n, 10000.0, device=DEV)


def _rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm())


@pytest.mark.parametrize("kind,hd,heads,kv", [("swiglu", 128, 4, 2), ("swiglu", 64, 6, 6), ("gelu", 128, 4, 1), ("moe", 64, 8, 2)])
@pytest.mark.parametrize("b,prompt", [(1, 1), (1, 9), (3, 100), (2, 333)])
def test_cached_block_matches_the_op_by_op_path(native_lib, monkeypatch, kind, hd, heads, kv, b, prompt):
    """Prompt into an empty cache, then two single tokens: outputs and caches of both paths (same inputs, each its own
    caches).  A handful of bf16 roundings apart: 2^-9 each over about ten tensors in a row."""
    from kempnerforge_b200.models import transformer
    from kempnerforge_b200.models.attention import KVCache

    block, cfg = _block(kind, hd, heads, kv)
    cos, sin = _tables(hd)
    xs = [_rand(b, n, cfg.dim, seed=11 + i) for i, n in enumerate((prompt, 1, 1))]
    runs = []
    for off in (False, True):
        monkeypatch.setattr(transformer, "_FUSED_BLOCK_OFF", off)
        cache = KVCache(b, prompt + 5, kv, hd, torch.bfloat16, torch.device(DEV))
        ys, at = [], 0
        with torch.no_grad():
            for x in xs:
                n = x.shape[1]
                ys.append(block(x, cos[at : at + n], sin[at : at + n], kv_cache=cache))
                at += n
        assert cache.seq_len == prompt + 2
        runs.append((ys, cache))
    assert native_lib.read_status() == 0
    for a, c in zip(*(r[0] for r in runs)):
        assert a.shape == c.shape and _rel(a, c) < 2e-2
    for name in ("k", "v"):
        got, want = (getattr(r[1], name) for r in runs)
        assert _rel(got, want) < 1e-2 and bool((got[:, prompt + 2 :] == 0).all())


@pytest.mark.parametrize("m", [1, 16, 17, 64])
@pytest.mark.parametrize("n,k", [(768, 768), (2304, 768), (768, 2048), (200, 72)])
def test_unsplit_products_equal_the_tile_kernel(native_lib, m, n, k):
    x, w = _rand(m, k, seed=1), _rand(n, k, seed=2)
    assert torch.equal(native_lib.gemm_rows(x, [w]), native_lib.gemm(x, w, mode=1))


@pytest.mark.parametrize("b,ctx", [(1, 1), (1, 300), (3, 77), (8, 1000), (20, 130)])
def test_small_models_keep_their_bits_when_decoding(native_lib, monkeypatch, b, ctx):
    """Head dim 64, weights below 8 MB: the fused step rounds where the separate ops round and sums in their order."""
    from kempnerforge_b200.models import transformer
    from kempnerforge_b200.models.attention import KVCache

    block, cfg = _block("swiglu", 64, 12, 12)
    cos, sin = _tables(64)
    x = _rand(b, 1, cfg.dim, seed=2)
    past = _rand(2, b, ctx, 12, 64, seed=3)
    out = []
    for off in (False, True):
        monkeypatch.setattr(transformer, "_FUSED_BLOCK_OFF", off)
        cache = KVCache(b, ctx + 4, 12, 64, torch.bfloat16, torch.device(DEV))
        cache.k[:, : ctx - 1], cache.v[:, : ctx - 1] = past[0, :, 1:], past[1, :, 1:]
        cache.seq_len = ctx - 1
        with torch.no_grad():
            out.append((block(x, cos[ctx - 1 : ctx], sin[ctx - 1 : ctx], kv_cache=cache), cache.k, cache.v))
    assert native_lib.read_status() == 0
    for a, c in zip(*out):
        assert torch.equal(a, c)


@pytest.mark.parametrize("kind,tokens", [("swiglu", (2, 333)), ("swiglu", (1, 20)), ("moe", (2, 200))])
def test_gradient_free_forward_matches_the_op_by_op_path(native_lib, monkeypatch, kind, tokens):
    from kempnerforge_b200.models import transformer

    block, cfg = _block(kind)
    cos, sin = _tables(128)
    x = _rand(*tokens, cfg.dim, seed=4)
    out = []
    for off in (False, True):
        monkeypatch.setattr(transformer, "_FUSED_BLOCK_OFF", off)
        with torch.no_grad():
            out.append(block(x, cos[: tokens[1]], sin[: tokens[1]]))
    assert native_lib.read_status() == 0 and _rel(*out) < 2e-2


def test_calls_the_gradient_free_path_does_not_cover_keep_their_behaviour(native_lib):
    """Hooks fire, a full cache raises and stays as it was, a prompt behind a non-empty cache and masks take the general path."""
    from kempnerforge_b200.models.attention import KVCache
    from kempnerforge_b200.ops import fused_infer

    block, cfg = _block("swiglu")
    cos, sin = _tables(128)
    x = _rand(2, 1, cfg.dim, seed=1)
    cache = KVCache(2, 2, 2, 128, torch.bfloat16, torch.device(DEV))
    seen = []
    hook = block.attention.register_forward_hook(lambda m, i, o: seen.append(o.shape))
    with torch.no_grad():
        block(x, cos[:1], sin[:1], kv_cache=cache)
    assert len(seen) == 1 and cache.seq_len == 1
    hook.remove()
    with torch.no_grad():
        assert fused_infer.run(block, _rand(2, 2, cfg.dim), cos, sin, cache) is None      # behind a non-empty cache
        assert fused_infer.run(block, x, cos.half(), sin.half(), cache) is None           # other tables
        block(x, cos[1:2], sin[1:2], kv_cache=cache)
        with pytest.raises(ValueError):
            block(x, cos[2:3], sin[2:3], kv_cache=cache)
    assert cache.seq_len == 2 and len(seen) == 1


@pytest.mark.parametrize("rows", [(4096, 1024, 1024), (768, 768, 768), (640, 128, 256)])
@pytest.mark.parametrize("s", [777, 300])
def test_rotary_projection_over_separate_weights(native_lib, rows, s):
    hd, k = 128, 1024
    x, ws = _rand(2 * s, k, scale=0.5, seed=1), [_rand(n, k, scale=0.5, seed=2 + i) for i, n in enumerate(rows)]
    ang = torch.arange(s, device=DEV)[:, None] * (10000.0 ** (-torch.arange(hd // 2, device=DEV) / (hd // 2)))
    cos, sin = ang.cos().float(), ang.sin().float()
    got = native_lib.qkv_rope(x, ws, cos, sin, s, hd)
    y = (x.double() @ torch.cat(ws).double().t()).view(2, s, -1, hd)
    mag = (x.double().abs() @ torch.cat(ws).double().abs().t()).view(2, s, -1, hd)
    lo, hi = y.chunk(2, -1)
    c, sn = cos.double()[None, :, None], sin.double()[None, :, None]
    rot = torch.cat([lo * c - hi * sn, hi * c + lo * sn], -1)
    n_rot = (rows[0] + rows[1]) // hd
    want = torch.cat([rot[:, :, :n_rot], y[:, :, n_rot:]], 2)
    swap = torch.cat(mag.chunk(2, -1)[::-1], -1)
    # small shapes round the projection before rotating: 2^-8 of both members of a pair
    assert native_lib.read_status() == 0
    assert bool(((got.double().view_as(want) - want).abs() <= 2.0**-7 * (y.abs() + torch.cat(y.abs().chunk(2, -1)[::-1], -1)) + 2.0**-15 * (mag + swap)).all())


@pytest.mark.parametrize("m,f,k", [(1554, 7168, 2048), (999, 2048, 768), (300, 640, 520)])
def test_swiglu_over_separate_weights_matches_the_stacked_one(native_lib, m, f, k):
    x, wg, wu = (_rand(n, k, scale=0.5, seed=i) for i, n in enumerate((m, f, f)))
    h, gu = native_lib.gemm_swiglu_pair(x, wg, wu)
    h2, gu2 = native_lib.gemm_swiglu(x, torch.cat([wg, wu]))
    assert native_lib.read_status() == 0 and torch.equal(h, h2) and torch.equal(gu, gu2)
    w = torch.cat([wg, wu])
    _check_dot(gu, x, w)


@pytest.mark.parametrize("b,s,hkv,hd,max_len,pad", [(1, 1, 1, 64, 1, 0), (2, 777, 8, 128, 800, 4096), (3, 33, 3, 64, 33, 192), (1, 257, 40, 128, 300, 0)])
def test_prompt_rows_into_both_caches(native_lib, b, s, hkv, hd, max_len, pad):
    """Bit for bit the strided copies, and nothing beyond the prompt."""
    width = hkv * hd
    rows = torch.randn(b * s, pad + 2 * width, device="cuda").bfloat16()
    k, v = (torch.full((b, max_len, hkv, hd), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    native_lib.cache_rows(rows[:, pad:], k, v, s)
    kv = rows[:, pad:].reshape(b, s, 2, hkv, hd)
    assert torch.equal(k[:, :s], kv[:, :, 0]) and torch.equal(v[:, :s], kv[:, :, 1])
    assert (k[:, s:] == 7).all() and (v[:, s:] == 7).all()
