"""Pair tiles cut to the number of tokens: every epilogue at ragged sizes against single-CTA tiles (the same sums, the same bits) and
the formulas."""

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


def _taken(kc, kind, m, n, k, hd=0):
    """Whether the product runs on tiles cut to its rows."""
    return kc.lib().kf_gemm_tokens_width(kind, m, n, k, hd, kc.sm_count()) > 0


@pytest.mark.parametrize("t,f,k", [(270, 1024, 512), (520, 14336, 256), (1554, 1408, 768), (777, 14336, 4096)])
def test_swiglu_and_its_gradient(native_lib, t, f, k):
    """Against a plain product on single-CTA tiles and the formulas on its rounded results."""
    kc = native_lib
    assert _taken(kc, 2, t, f, k) and _taken(kc, 4, t, f, k)
    x, wg, wu = _rand(t, k, seed=1), _rand(f, k, scale=k**-0.5, seed=2), _rand(f, k, scale=k**-0.5, seed=3)
    h, gu = kc.gemm_swiglu_pair(x, wg, wu)
    only, none = kc.gemm_swiglu_pair(x, wg, wu, want_gu=False)
    assert none is None and torch.equal(h, only) and torch.equal(gu, kc.gemm(x, torch.cat([wg, wu]), mode=1))
    g, u = gu[:, :f].double(), gu[:, f:].double()
    sig = g.sigmoid()
    want = g * sig * u
    # fp32 with the fast exponential and division (below 2^-19 each), then one rounding to bf16
    assert bool(((h.double() - want).abs() <= 2.0**-8 * want.abs()).all())
    dy, wd = _rand(t, k, seed=4), _rand(k, f, scale=k**-0.5, seed=5)
    dh = kc.gemm(dy, wd, b_kmajor=False, mode=1).double()
    dg, du = dh * u * sig * (1 + g * (1 - sig)), dh * g * sig
    got = kc.gemm_swiglu_bwd(dy, wd, gu).double()
    assert kc.read_status() == 0
    # dg vanishes where g (1 - sig) is -1: the bound is relative to the sum of the magnitudes there
    assert bool(((got[:, f:] - du).abs() <= 2.0**-8 * du.abs()).all())
    mag = (dh * u * sig).abs() * (1 + (g * (1 - sig)).abs())
    assert bool(((got[:, :f] - dg).abs() <= 2.0**-8 * dg.abs() + 2.0**-18 * mag).all())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("seqs,s,heads,kv,k", [(1, 300, 12, 6, 256), (3, 518, 32, 8, 512), (3, 259, 16, 4, 768), (1, 1000, 6, 2, 64)])
def test_rotation(native_lib, seqs, s, heads, kv, k, hd):
    """Against the product and the rotation in 64 bits; the position starts over with every sequence."""
    kc = native_lib
    ws = [_rand(n * hd, k, scale=k**-0.5, seed=2 + i) for i, n in enumerate((heads, kv, kv))]
    x, n, rope_cols = _rand(seqs * s, k, seed=1), (heads + 2 * kv) * hd, (heads + kv) * hd
    assert _taken(kc, 3, seqs * s, n, k, hd)
    ang = torch.rand(s, hd // 2, device=DEV, generator=torch.Generator(device=DEV).manual_seed(5)) * 6.0
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()

    def run(weights):
        out = torch.empty(x.shape[0], n, dtype=torch.bfloat16, device=DEV)
        ptrs, counts, _ = kc._weights3(weights)
        kc._check(kc.lib().kf_gemm_rope_bf16(x.data_ptr(), *ptrs, out.data_ptr(), x.shape[0], *counts, k, k, k, n, cos.data_ptr(),
                                             sin.data_ptr(), s, rope_cols, hd, kc.sm_count(), kc._stream()), "rope")
        return out

    got = run(ws)
    assert torch.equal(got, run([torch.cat(ws)])) and kc.read_status() == 0
    w = torch.cat(ws)
    assert torch.equal(got[:, rope_cols:], kc.gemm(x, w, mode=1)[:, rope_cols:])
    c, sn = (t.double().repeat(seqs, 1)[:, None] for t in (cos, sin))

    def rotated(y):
        a, b = y[:, :rope_cols].view(-1, heads + kv, hd).split(hd // 2, -1)
        return torch.cat([a * c - b * sn, b * c + a * sn], -1).reshape(-1, rope_cols)

    want = rotated(x.double() @ w.double().t())
    c, sn = c.abs(), sn.abs()
    a, b = (x.double().abs() @ w.double().abs().t())[:, :rope_cols].view(-1, heads + kv, hd).split(hd // 2, -1)
    mag = torch.cat([a * c + b * sn, b * c + a * sn], -1).reshape(-1, rope_cols)
    # fp32 sums in any order and the rotation (2^-16 of the magnitudes), one rounding to bf16
    assert bool(((got[:, :rope_cols].double() - want).abs() <= 2.0**-8 * want.abs() + 2.0**-16 * mag).all())


@pytest.mark.parametrize("t,k,rows", [(300, 768, (768, 768, 768)), (1554, 4096, (4096, 1024, 1024)), (2999, 2048, (1408, 1408)), (700, 520, (64, 72))])
def test_input_gradient_of_stacked_weights(native_lib, t, k, rows):
    kc = native_lib
    assert _taken(kc, 1, t, k, sum(rows)) == (t == 1554)   # the others take the single-CTA tiles, which read the stack as well
    ws = [_rand(n, k, scale=0.1, seed=2 + i) for i, n in enumerate(rows)]
    dy = _rand(t, sum(rows), seed=1)
    assert torch.equal(kc.dgrad_rows(dy, ws), kc.gemm(dy, torch.cat(ws), b_kmajor=False, mode=1))
    assert kc.read_status() == 0
