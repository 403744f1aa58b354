"""RMSNorm on both sides of every line of its dispatch: rows per warp or block, words held per thread, rows longer than what is held."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("d", [8, 768, 1024, 1032, 2048, 2056, 4096, 4104, 8192, 8200])
@pytest.mark.parametrize("rows", [1, 1023, 1024, 1309])
def test_against_double(native_lib, rows, d):
    torch.manual_seed(d)
    x, dy, res = (torch.randn(rows, d, device=DEV).bfloat16() for _ in range(3))
    w = (1 + 0.1 * torch.randn(d, device=DEV)).bfloat16()
    y, rstd = native_lib.rmsnorm_fwd(x, w, 1e-5)
    xd, g = x.double(), dy.double() * w.double()
    r = (xd.square().mean(-1, keepdim=True) + 1e-5).rsqrt()
    assert torch.allclose(rstd.double(), r[:, 0], rtol=2.0**-18)             # fp32 sums of d squares
    want = xd * r * w.double()
    assert ((y.double() - want).abs() <= want.abs() * 2.0**-8).all()         # one rounding to bf16
    first, second = r * g, xd * r**3 * (g * xd).mean(-1, keepdim=True)
    for residual, out in ((None, None), (res, None), (res.clone(), "residual"), (res, "dy")):
        dyi = dy.clone()
        target = {None: None, "residual": residual, "dy": dyi}[out]
        dx, _ = native_lib.rmsnorm_bwd(dyi, x, w, rstd, residual_grad=residual, out=target)
        add = res.double() if residual is not None else torch.zeros_like(first)
        # the sum is rounded to bf16; its terms are right to 2^-18, the mean's to that of the magnitudes it adds up
        err = 2.0**-17 * (first.abs() + (xd * r**3).abs() * (g * xd).abs().mean(-1, keepdim=True) + add.abs())
        total = first - second + add
        assert ((dx.double() - total).abs() <= total.abs() * 2.0**-8 + err).all()
