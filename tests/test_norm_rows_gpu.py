"""RMSNorm at the edges of the warp-per-row kernels (rows 1024 and up, widths up to 4096) and of the column sums."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,d", [(1023, 768), (1024, 8), (1025, 256), (1027, 1024), (1030, 1032), (2000, 2048), (1024, 2056), (1500, 1032), (1100, 2048),
                                    (4097, 4096), (1024, 4104), (3, 4096), (149, 40)])
@pytest.mark.parametrize("alias", [False, True])
def test_norm_forward_and_backward(native_lib, rows, d, alias):
    g = torch.Generator(device="cuda").manual_seed(rows + d)
    x, dy, res = (torch.randn(rows, d, device="cuda", generator=g).bfloat16() for _ in range(3))
    w = (1 + 0.1 * torch.randn(d, device="cuda", generator=g)).bfloat16()
    y, rstd = native_lib.rmsnorm_fwd(x, w, 1e-5)
    xd, wd, gd = x.double(), w.double(), dy.double()
    r = torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5)
    want = xd * r * wd
    # one rounding to bf16 (half an ulp: up to 2^-8 of the value), fp32 mean of squares and reciprocal root (2^-18 together)
    assert bool(((y.double() - want).abs() <= (2.0**-8 + 2.0**-18) * want.abs()).all())
    assert bool(((rstd.double() - r[:, 0]).abs() <= 2.0**-18 * r[:, 0]).all())
    out = dy.clone() if alias else None
    dx, dw = native_lib.rmsnorm_bwd(out if alias else dy, x, w, rstd, residual_grad=res, out=out)
    gw = gd * wd
    wdx = res.double() + r * gw - xd * r**3 * (gw * xd).mean(-1, keepdim=True)
    mag = res.double().abs() + r * gw.abs() + xd.abs() * r**3 * (gw * xd).abs().mean(-1, keepdim=True)
    assert bool(((dx.double() - wdx).abs() <= 2.0**-8 * wdx.abs() + 2.0**-16 * mag).all())
    wdw, mdw = (gd * xd * r).sum(0), (gd * xd * r).abs().sum(0)
    assert bool(((dw.double() - wdw).abs() <= 2.0**-8 * wdw.abs() + 2.0**-16 * mdw).all())
