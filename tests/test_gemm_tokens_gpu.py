"""Pair tiles cut to the number of tokens: every epilogue at ragged sizes against the tiles of 256 rows (the same sums, the same bits)."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _rand(*shape, scale=1.0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, device=DEV, generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("w_mn", [False, True])
@pytest.mark.parametrize("t,f,k", [(1, 8, 64), (31, 264, 72), (33, 256, 768), (255, 40, 136), (257, 520, 200), (300, 4096, 512),
                                   (777, 1000, 64), (1554, 4096, 1024), (2500, 776, 256)])
def test_plain(native_lib, t, f, k, w_mn):
    kc = native_lib
    x = _rand(t, k + 8, seed=1)[:, :k]
    w = _rand(k, f + 16, seed=2)[:, :f] if w_mn else _rand(f, k + 16, seed=2)[:, :k]
    res = _rand(t, f + 8, seed=3)[:, :f]
    frame = torch.full((t + 1, f + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    kc.gemm(x, w, b_kmajor=not w_mn, out=frame[:t, :f], mode=3)
    got = kc.gemm(x, w, b_kmajor=not w_mn, residual=res, mode=3)
    assert kc.read_status() == 0
    assert torch.equal(frame[:t, :f], kc.gemm(x, w, b_kmajor=not w_mn, mode=1))
    assert torch.equal(got, kc.gemm(x, w, b_kmajor=not w_mn, residual=res, mode=1))
    assert bool((frame[t:] == 7).all()) and bool((frame[:, f:] == 7).all())


def _padded(x):
    """The same rows and zeros up to the next multiple of 256, where the 256-row tiles are taken."""
    t = x.shape[0]
    return torch.cat([x, x.new_zeros(-t % 256, x.shape[1])])


@pytest.mark.parametrize("t,f,k", [(270, 1024, 512), (520, 14336, 256), (1554, 1408, 768), (777, 14336, 4096)])
def test_swiglu_and_its_gradient(native_lib, t, f, k):
    kc = native_lib
    x, wg, wu = _rand(t, k, seed=1), _rand(f, k, scale=k**-0.5, seed=2), _rand(f, k, scale=k**-0.5, seed=3)
    h, gu = kc.gemm_swiglu_pair(x, wg, wu)
    only, none = kc.gemm_swiglu_pair(x, wg, wu, want_gu=False)
    hp, gup = kc.gemm_swiglu_pair(_padded(x), wg, wu)
    assert none is None and torch.equal(h, only) and torch.equal(h, hp[:t]) and torch.equal(gu, gup[:t])
    dy, wd = _rand(t, k, seed=4), _rand(k, f, scale=k**-0.5, seed=5)
    want = kc.gemm_swiglu_bwd(_padded(dy), wd, gup.clone())[:t]
    assert torch.equal(kc.gemm_swiglu_bwd(dy, wd, gu), want)
    assert kc.read_status() == 0


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("seqs,s,heads,kv,k", [(1, 300, 12, 6, 256), (3, 518, 32, 8, 512), (3, 259, 16, 4, 768), (1, 1000, 6, 2, 64)])
def test_rotation(native_lib, seqs, s, heads, kv, k, hd):
    kc = native_lib
    ws = [_rand(n * hd, k, scale=k**-0.5, seed=2 + i) for i, n in enumerate((heads, kv, kv))]
    x, n, rope_cols = _rand(seqs * s, k, seed=1), (heads + 2 * kv) * hd, (heads + kv) * hd
    ang = torch.rand(s + 256, hd // 2, device=DEV, generator=torch.Generator(device=DEV).manual_seed(5)) * 6.0
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()

    def run(rows, weights, length):
        out = torch.empty(rows.shape[0], n, dtype=torch.bfloat16, device=DEV)
        ptrs, counts, _ = kc._weights3(weights)
        kc._check(kc.lib().kf_gemm_rope_bf16(rows.data_ptr(), *ptrs, out.data_ptr(), rows.shape[0], *counts, k, k, k, n, cos.data_ptr(),
                                             sin.data_ptr(), length, rope_cols, hd, kc.sm_count(), kc._stream()), "rope")
        return out

    got = run(x, ws, s)
    assert torch.equal(got, run(x, [torch.cat(ws)], s))
    for i in range(seqs):   # the position starts over with every sequence
        part = x[i * s : (i + 1) * s]
        assert torch.equal(got[i * s : (i + 1) * s], run(_padded(part), ws, s + 256)[:s])
    assert kc.read_status() == 0


@pytest.mark.parametrize("t,k,rows", [(300, 768, (768, 768, 768)), (1554, 4096, (4096, 1024, 1024)), (2999, 2048, (1408, 1408)), (700, 520, (64, 72))])
def test_input_gradient_of_stacked_weights(native_lib, t, k, rows):
    kc = native_lib
    ws = [_rand(n, k, scale=0.1, seed=2 + i) for i, n in enumerate(rows)]
    dy = _rand(t, sum(rows), seed=1)
    assert torch.equal(kc.dgrad_rows(dy, ws), kc.gemm(dy, torch.cat(ws), b_kmajor=False, mode=1))
    assert kc.read_status() == 0
