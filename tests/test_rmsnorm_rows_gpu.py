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


@pytest.mark.parametrize("rows,d", [(1024, 256), (1024, 1024), (1025, 2048), (1024, 4096), (1554, 4096)])
def test_the_squares_of_many_rows_are_added_in_one_order(native_lib, rows, d):
    """A warp per row, lane l the 16-byte words l, l + 32, ..., then the lanes in pairs 16, 8, 4, 2, 1 apart: a step through several
    blocks turns other last bits of rstd into outputs that differ like independent roundings.  (Powers of two: the mean is exact.)"""
    torch.manual_seed(rows + d)
    x = torch.randn(rows, d, device=DEV).bfloat16()
    _, rstd = native_lib.rmsnorm_fwd(x, torch.ones(d, device=DEV).bfloat16(), 1e-5)
    words = x.float().view(rows, -1, 32, 8)
    ss = torch.zeros(rows, 32, device=DEV)
    for c in range(words.shape[1]):
        for i in range(8):
            ss = ss + words[:, c, :, i] ** 2   # the square of a bf16 value is exact in fp32
    lane = torch.arange(32, device=DEV)
    for o in (16, 8, 4, 2, 1):
        ss = ss + ss[:, lane ^ o]
    assert torch.equal(rstd, (ss[:, 0] / d + 1e-5).rsqrt())
