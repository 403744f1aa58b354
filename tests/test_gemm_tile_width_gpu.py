"""CTA-pair GEMMs over the tile widths the launch picks (128 to 256 columns), ragged edges included, against fp64 products."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _rand(*shape, seed):
    return (torch.randn(*shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed)) * 0.5).bfloat16()


def _check(got, want, mag):
    # one bf16 rounding (half an ulp, up to 2^-8 relative) of an fp32 sum in any order
    assert bool(((got.double() - want).abs() <= 2.0**-8 * want.abs() + 2.0**-16 * mag).all())


# one round of narrow tiles; 224 wide (7 x 19 and 12 x 23 tiles); 256; just past a round; widths that end inside a chunk
SHAPES = [(999, 768, 768), (300, 2304, 768), (1554, 4096, 520), (3000, 5120, 264), (2047, 4096, 200), (256, 19200, 136),
          (257, 8, 64), (512, 4728, 320), (1024, 200, 1000)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("a_k,b_k", [(True, True), (True, False), (False, False)])
def test_every_tile_width_matches_fp64_and_stays_inside_its_output(native_lib, m, n, k, a_k, b_k):
    if not a_k:
        m += -m % 8
    a, b = _rand(m, k, seed=1), _rand(n, k, seed=2)
    want, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    ai, bi = a if a_k else a.t().contiguous(), b if b_k else b.t().contiguous()
    frame = torch.full((m + 1, n + 8), 5.0, dtype=torch.bfloat16, device=DEV)
    got = native_lib.gemm(ai, bi, a_kmajor=a_k, b_kmajor=b_k, mode=2, out=frame[:m, :n])
    assert native_lib.read_status() == 0
    _check(got, want, mag)
    assert bool((frame[m:] == 5).all()) and bool((frame[:, n:] == 5).all())
    # the sums over K have one order whatever the tile: the single-CTA kernel gives the same bits
    assert torch.equal(got, native_lib.gemm(ai, bi, a_kmajor=a_k, b_kmajor=b_k, mode=1))


def test_residual_accumulation_and_fp32_output(native_lib):
    m, n, k = 1554, 4096, 520
    a, b, r = _rand(m, k, seed=1), _rand(n, k, seed=2), _rand(m, n, seed=3)
    want, mag = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    _check(native_lib.gemm(a, b, residual=r, mode=2), want + r.double(), mag + r.double().abs())
    out = r.float()
    native_lib.gemm(a, b, out=out, accumulate=True, mode=2)
    assert bool(((out.double() - want - r.double()).abs() <= 2.0**-16 * (mag + r.double().abs())).all())


@pytest.mark.parametrize("m,f,k", [(1554, 4096, 128), (300, 200, 64), (999, 2048, 768)])
def test_swiglu_gradient_epilogue_over_narrow_tiles(native_lib, m, f, k):
    dy, w, gu = _rand(m, k, seed=1), _rand(k, f, seed=2), _rand(m, 2 * f, seed=3)
    got = native_lib.gemm_swiglu_bwd(dy, w, gu.clone())
    dh = native_lib.gemm(dy, w, b_kmajor=False)          # the epilogue rounds dh to bf16, like two kernels
    g, u = gu[:, :f].double(), gu[:, f:].double()
    s = torch.sigmoid(g)
    want = torch.cat([dh.double() * u * s * (1 + g * (1 - s)), dh.double() * g * s], 1)
    assert native_lib.read_status() == 0
    # fast exponential and division (2^-20), one rounding
    assert bool(((got.double() - want).abs() <= 2.0**-8 * want.abs() + 2.0**-18 * dh.double().abs().repeat(1, 2)).all())
