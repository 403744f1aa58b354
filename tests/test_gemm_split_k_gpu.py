"""Products over a long reduction that are cut along K, at the edges of tiles and pieces, against fp64 and the whole product."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("m,n,k", [(1, 8, 8192), (100, 264, 8200), (257, 768, 12296), (333, 1024, 33000), (1300, 2056, 16392)])
def test_pieces_match_fp64_and_stay_inside_the_output(native_lib, m, n, k):
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    a = (torch.randn(m, k, device=DEV, generator=g) * 0.5).bfloat16()
    b = (torch.randn(k, n, device=DEV, generator=g) * 0.5).bfloat16()
    assert native_lib.lib().kf_gemm_k_pieces(m, n, k, native_lib.sm_count()) > 1
    frame = torch.full((m + 1, n + 8), 5.0, dtype=torch.bfloat16, device=DEV)
    got = native_lib.gemm(a, b, b_kmajor=False, out=frame[:m, :n])
    assert native_lib.read_status() == 0
    want, mag = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    # one bf16 rounding (half an ulp, up to 2^-8 relative) of an fp32 sum in any order
    assert bool(((got.double() - want).abs() <= 2.0**-8 * want.abs() + 2.0**-16 * mag).all())
    assert bool((frame[m:] == 5).all()) and bool((frame[:, n:] == 5).all())
    assert torch.equal(got, native_lib.gemm(a, b, b_kmajor=False))                       # fixed order of the pieces
    whole = native_lib.gemm(a, b, b_kmajor=False, mode=1)
    err, ref = ((x.double() - want).norm() for x in (got, whole))
    assert float(err) <= 1.05 * float(ref)                  # no less precise than the product in one piece
    # what the split does not cover stays on the whole product
    f32 = native_lib.gemm(a, b, b_kmajor=False, out_dtype=torch.float32)
    assert bool(((f32.double() - want).abs() <= 2.0**-16 * mag).all())
