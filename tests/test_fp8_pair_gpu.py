"""The fp8 product on CTA pairs at the edges of its tiles (128 to 256 columns, 256 rows), against fp64."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


# one row; narrow tiles; past a row of tiles and inside a 16-byte step of K; 224 columns (8 x 64 tiles); 256; several rounds
@pytest.mark.parametrize("m,n,k", [(1, 16, 16), (1, 4096, 512), (129, 136, 144), (257, 200, 2064), (2000, 14336, 272),
                                   (300, 768, 768), (4096, 4736, 128), (14336, 2048, 2000)])
@pytest.mark.parametrize("e5m2", [False, True])
def test_every_tile_width_matches_fp64_and_stays_inside_its_output(native_lib, m, n, k, e5m2):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    a, b = (torch.randn(r, k, device=DEV, generator=g).bfloat16() for r in (m, n))
    sa, sb = native_lib.fp8_scale(a, e5m2), native_lib.fp8_scale(b)
    a8, b8 = native_lib.fp8_cast(a, sa, e5m2)[0], native_lib.fp8_cast(b, sb, False)[0]
    frame = torch.full((m + 1, n + 8), 5.0, dtype=torch.bfloat16, device=DEV)
    got = native_lib.gemm_fp8(a8, b8, sa, sb, e5m2, False, out=frame[:m, :n])
    assert native_lib.read_status() == 0
    ad = a8.view(torch.float8_e5m2 if e5m2 else torch.float8_e4m3fn).float().double()
    bd = b8.view(torch.float8_e4m3fn).float().double()
    scale = (sa * sb).double()
    want, mag = ad @ bd.t() / scale, ad.abs() @ bd.abs().t() / scale
    # a sum of k exact products, each addition off by at most 2^-23 of the partial sum, then one bf16 rounding (2^-8)
    bound = 2.0**-8 * want.abs() + k * 2.0**-23 * mag
    assert bool(((got.double() - want).abs() <= bound).all())
    assert bool((frame[m:] == 5).all()) and bool((frame[:, n:] == 5).all())
    acc = native_lib.gemm_fp8(a8, b8, sa, sb, e5m2, False, out=got.clone(), accumulate=True)
    assert bool(((acc.double() - want - got.double()).abs() <= bound + 2.0**-8 * (want + got.double()).abs()).all())
