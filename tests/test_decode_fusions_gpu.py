"""Projections of a generation step that take the norm and the rotation along: bit for bit the separate kernels, except that the
rotation of heads of 128 rounds the second half of a pair in another place."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _rand(*shape, scale=1.0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, device=DEV, generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("m,f,k", [(1, 64, 8), (1, 200, 72), (2, 2048, 768), (3, 136, 2056), (4, 14336, 4096), (4, 1024, 5120), (1, 64, 9000)])
def test_norm_along_with_swiglu(native_lib, m, f, k):
    kc, L = native_lib, native_lib.lib()
    assert m <= L.kf_skinny_norm_rows()
    x = _rand(m + 1, k + 8, scale=3.0, seed=1)[:m, :k]                       # a row pitch of its own
    gain, wg, wu = 1 + 0.1 * _rand(k, seed=2), _rand(f, k, scale=k**-0.5, seed=3), _rand(f, k, scale=k**-0.5, seed=4)
    n, _ = kc.rmsnorm_fwd(x.contiguous(), gain, 1e-5)
    out = []
    for src, g in ((n, None), (x, gain.data_ptr())):
        h = torch.empty(m, f, dtype=torch.bfloat16, device=DEV)
        kc._check(L.kf_gemm_skinny_norm_swiglu_bf16(src.data_ptr(), g, 1e-5, wg.data_ptr(), wu.data_ptr(), h.data_ptr(), m, f, k,
                                                    src.stride(0), k, k, f, 0, kc.sm_count(), kc._stream()), "swiglu")
        out.append(h)
    assert native_lib.read_status() == 0
    assert torch.equal(*out)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("b,heads,kv,k", [(1, 12, 12, 768), (2, 3, 1, 264), (4, 16, 4, 2048), (5, 6, 3, 520), (9, 4, 2, 768), (16, 6, 2, 3616),
                                            (33, 4, 2, 768)])
def test_projection_rotation_and_cache(native_lib, b, heads, kv, k, hd):
    kc, L = native_lib, native_lib.lib()
    qc, kvc = heads * hd, kv * hd
    x, gain = _rand(b, k, seed=1), 1 + 0.1 * _rand(k, seed=2)
    ws = [_rand(n, k, scale=k**-0.5, seed=3 + i) for i, n in enumerate((qc, kvc, kvc))]
    ang = torch.rand(1, hd // 2, device=DEV, generator=torch.Generator(device=DEV).manual_seed(9)) * 6.0
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    n, _ = kc.rmsnorm_fwd(x, gain, 1e-5)
    qkv = kc.gemm_rows(n, ws).view(b, 1, heads + 2 * kv, hd)
    x2 = qkv[..., hd // 2 :].clone()
    x1 = qkv[..., : hd // 2].clone()
    kc.rope(qkv, cos, sin, heads + kv, inverse=False, out=qkv)
    if hd == 128:   # the second half of a pair: x1 sin in full precision, x2 cos rounded to fp32, their sum rounded once
        hi = (x1.double() * sin.double() + (x2.double() * cos.double()).float().double()).float().bfloat16()
        qkv[:, :, : heads + kv, hd // 2 :] = hi[:, :, : heads + kv]
    want = qkv.view(b, -1).split([qc, kvc, kvc], 1)
    for src, g in ((n, None), (x, gain.data_ptr())) if b <= L.kf_skinny_norm_rows() else ((n, None),):
        q = torch.empty(b, qc, dtype=torch.bfloat16, device=DEV)
        cache = torch.full((2, b, 3, kvc), 7.0, dtype=torch.bfloat16, device=DEV)
        kc._check(L.kf_gemm_skinny_norm_qkv_bf16(src.data_ptr(), g, 1e-5, *(w.data_ptr() for w in ws), q.data_ptr(),
                                                 cache[0, 0, 1].data_ptr(), cache[1, 0, 1].data_ptr(), b, 1, k, qc, kvc, hd, k, k, k, k, qc,
                                                 3 * kvc, cos.data_ptr(), sin.data_ptr(), 0, kc.sm_count(), kc._stream()), "qkv")
        assert native_lib.read_status() == 0
        for got, w in zip((q, cache[0, :, 1], cache[1, :, 1]), want):
            assert torch.equal(got, w)
        assert bool((cache[:, :, 0] == 7).all()) and bool((cache[:, :, 2] == 7).all())
    assert L.kf_gemm_skinny_norm_qkv_bf16(x.data_ptr(), gain.data_ptr(), 1e-5, *(w.data_ptr() for w in ws), q.data_ptr(),
                                          cache.data_ptr(), cache.data_ptr(), L.kf_skinny_norm_rows() + 1, 1, k, qc, kvc, hd, k, k, k, k,
                                          qc, 3 * kvc, cos.data_ptr(), sin.data_ptr(), 0, kc.sm_count(), kc._stream()) == 5


@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 16])
@pytest.mark.parametrize("rows,k", [([8], 32), ([768], 768), ([24, 40, 8], 96), ([768], 2048), ([256, 64], 1504), ([512], 4096),
                                    ([136], 3616), ([64], 4800)])
def test_small_weights_keep_the_bits_of_the_tile_kernel(native_lib, m, rows, k):
    kc = native_lib
    x = _rand(m, k + 8, seed=1)[:, :k]
    ws = [_rand(n, k + 16, scale=0.3, seed=2 + i)[:, :k] for i, n in enumerate(rows)]
    res = _rand(m, sum(rows), seed=7)
    frame = torch.full((m + 1, sum(rows) + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    out = kc._stream_rows(x, ws, None, frame[:m, : sum(rows)])
    with_res = kc._stream_rows(x, ws, res, None)
    assert kc.read_status() == 0
    w = torch.cat(ws)
    assert torch.equal(out, kc.gemm(x, w, mode=1)) and torch.equal(with_res, kc.gemm(x, w, residual=res, mode=1))
    assert bool((frame[m:] == 7).all()) and bool((frame[:, sum(rows):] == 7).all())


@pytest.mark.parametrize("m", [1, 4, 8, 9, 15, 16])
@pytest.mark.parametrize("f,k", [(8, 32), (2048, 768), (136, 3616), (64, 4608)])
def test_small_weights_with_swiglu_against_the_tile_kernel(native_lib, m, f, k):
    """Gate and up on single-CTA tiles, then the SwiGLU kernel; with the norm along, the norm kernel first."""
    kc, L = native_lib, native_lib.lib()
    x, gain = _rand(m, k, scale=2.0, seed=1), 1 + 0.1 * _rand(k, seed=2)
    wg, wu = _rand(f, k, scale=k**-0.5, seed=3), _rand(f, k, scale=k**-0.5, seed=4)
    w = torch.cat([wg, wu])
    frame = torch.full((m + 1, f + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    for g in (None, gain) if m <= L.kf_skinny_norm_rows() else (None,):
        n = x if g is None else kc.rmsnorm_fwd(x, g, 1e-5)[0]
        kc._check(L.kf_gemm_skinny_norm_swiglu_bf16(x.data_ptr(), kc._ptr(g), 1e-5, wg.data_ptr(), wu.data_ptr(), frame.data_ptr(), m, f, k,
                                                    k, k, k, f + 8, 0, kc.sm_count(), kc._stream()), "swiglu")
        assert native_lib.read_status() == 0
        assert torch.equal(frame[:m, :f], kc.swiglu_fwd(kc.gemm(n, w, mode=1)))
    assert bool((frame[m:] == 7).all()) and bool((frame[:, f:] == 7).all())


def _model(heads, kv, batch, ctx, layers=3, **over):
    from kempnerforge_b200.config import ModelConfig
    from kempnerforge_b200.models.attention import KVCache
    from kempnerforge_b200.models.transformer import Transformer

    torch.manual_seed(0)
    cfg = ModelConfig(dim=512, n_layers=layers, n_heads=heads, n_kv_heads=kv, vocab_size=256, ffn_hidden_dim=768, max_seq_len=512, **over)
    model = Transformer(cfg).to(DEV, torch.bfloat16).eval()
    model._rope_cos = model._rope_sin = None
    caches = [KVCache(batch, ctx + 8, kv, 512 // heads, torch.bfloat16, torch.device(DEV)) for _ in range(layers)]
    for i, c in enumerate(caches):
        c.k.copy_(_rand(*c.k.shape, seed=20 + i))
        c.v.copy_(_rand(*c.v.shape, seed=40 + i))
        c.seq_len = ctx
    return model, caches


def _steps(model, caches, batch, n=3):
    start = [(c.k.clone(), c.v.clone(), c.seq_len) for c in caches]
    tokens = torch.arange(batch, device=DEV)[:, None] % 256
    with torch.no_grad():
        out = [model(tokens + i, kv_caches=caches) for i in range(n)]
    out += [t.clone() for c in caches for t in (c.k, c.v)] + [c.seq_len for c in caches]
    for c, (k, v, length) in zip(caches, start):
        c.k.copy_(k)
        c.v.copy_(v)
        c.seq_len = length
    return out


@pytest.mark.parametrize("heads,kv,batch,ctx", [(8, 8, 1, 1), (8, 2, 1, 130), (4, 4, 1, 200), (4, 2, 3, 77), (4, 2, 6, 64)])
def test_all_blocks_in_one_call(native_lib, monkeypatch, heads, kv, batch, ctx):
    from kempnerforge_b200.ops import fused_infer

    model, caches = _model(heads, kv, batch, ctx)
    used, native = [], fused_infer.run_layers
    monkeypatch.setattr(fused_infer, "run_layers", lambda *a: used.append(native(*a)) or used[-1])
    got = _steps(model, caches, batch)
    assert len(used) == 3 and all(u is not None for u in used) and native_lib.read_status() == 0
    monkeypatch.setattr(fused_infer, "run_layers", lambda *a: None)
    want = _steps(model, caches, batch)
    assert all(torch.equal(a, b) if torch.is_tensor(a) else a == b for a, b in zip(got, want))


def test_models_that_go_block_by_block(native_lib):
    from kempnerforge_b200.ops import fused_infer

    def run(model, caches, batch=1):
        x = _rand(batch, 1, 512)
        cos, sin = model.rope_tables(x.device, min(c.seq_len for c in caches), 1)
        with torch.no_grad():
            return fused_infer.run_layers(list(model.layers.values()), x, cos, sin, caches)

    model, caches = _model(8, 8, 1, 40)
    assert run(model, caches) is not None and [c.seq_len for c in caches] == [41] * 3
    caches[2].seq_len = caches[2].k.size(1)                                     # full: the error comes from the cache itself
    assert run(model, caches) is None and [c.seq_len for c in caches[:2]] == [41] * 2
    assert run(model, [caches[0]] * 3) is None and run(model, caches[:2]) is None
    handle = model.layers["1"].register_forward_hook(lambda m, a, o: o)
    caches[2].seq_len = 41
    assert run(model, caches) is None
    handle.remove()
    assert run(model, caches) is not None
    assert run(*_model(8, 8, 2, 40), batch=2) is None                           # heads of 64, several sequences: the library's attention
    assert run(*_model(4, 4, 1, 40, qk_norm=True)) is None


@pytest.mark.parametrize("written", ["weight", "gain", "tables"])
@pytest.mark.parametrize("dim,heads,kv,ffn,batch", [(768, 12, 12, 2048, 1), (512, 4, 2, 768, 4), (512, 4, 2, 768, 6), (4096, 32, 8, 4096, 1)])
def test_operands_written_by_the_kernel_before_the_step(native_lib, dim, heads, kv, ffn, batch, written):
    """The kernel in front of a generation step may have written any operand of its first projection."""
    from kempnerforge_b200.config import ModelConfig
    from kempnerforge_b200.models.attention import KVCache
    from kempnerforge_b200.models.transformer import TransformerBlock

    torch.manual_seed(0)
    cfg = ModelConfig(dim=dim, n_layers=1, n_heads=heads, n_kv_heads=kv, vocab_size=64, ffn_hidden_dim=ffn, max_seq_len=256)
    block = TransformerBlock(cfg, 0).to(DEV, torch.bfloat16).eval()
    hd, ctx = dim // heads, 100
    cache = KVCache(batch, 128, kv, hd, torch.bfloat16, torch.device(DEV))
    for i, t in enumerate((cache.k, cache.v)):
        t.copy_(_rand(*t.shape, seed=20 + i))
    x, tables = _rand(batch, 1, dim, seed=1), torch.zeros(2, 1, hd // 2, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(3)
    if written == "tables":
        target = tables
        versions = [torch.rand(2, 1, hd // 2, device=DEV, generator=g) for _ in range(2)]
    else:
        target = block.attention.v_proj.weight if written == "weight" else block.attention_norm.weight
        versions = [_rand(*target.shape, scale=0.05, seed=5 + i) for i in range(2)]

    def step(sync):
        cache.seq_len = ctx
        if sync:
            torch.cuda.synchronize()
        y = block(x, tables[0], tables[1], kv_cache=cache)
        return [y, cache.k[:, ctx].clone(), cache.v[:, ctx].clone()]

    with torch.no_grad():
        want = []
        for v in versions:
            target.copy_(v)
            want.append(step(sync=True))
        assert not all(torch.equal(a, b) for a, b in zip(*want))
        got = []
        for i in range(40):
            target.copy_(versions[i & 1])
            got.append(step(sync=False))
    assert native_lib.read_status() == 0
    assert all(torch.equal(a, b) for i, out in enumerate(got) for a, b in zip(out, want[i & 1]))
