"""Cross entropy whose row maxima and sums come from the product that writes the logits."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


# Columns: a last tile of 8, 16, 24 and 136 columns; rows: a block of 32 that is not full, tiles of 256 that are not
@pytest.mark.parametrize("rows,v,k", [(2047, 128256, 64), (4096, 9224, 128), (1001, 32024, 64), (768, 50312, 72), (8200, 4104, 64), (2560, 9232, 256)])
def test_against_double(native_lib, monkeypatch, rows, v, k):
    cu = native_lib
    monkeypatch.setattr(cu, "LOGITS_MIN_K", 0)
    monkeypatch.setattr(cu, "LOGITS_MIN_BYTES", 0)
    torch.manual_seed(v)
    h, w = torch.randn(rows, k, device=DEV).bfloat16(), torch.randn(v, k, device=DEV).mul_(3 * k**-0.5).bfloat16()
    h[1] = 0            # equal logits
    h[2] *= 30          # a row whose largest logit takes (nearly) all
    logits, tiles = cu.gemm_logits(h, w)
    assert tiles is not None and torch.equal(logits, cu.gemm(h, w))
    labels = torch.randint(0, v, (rows,), device=DEV)
    labels[0], labels[1], labels[3], labels[4::7] = 0, v - 1, v, -100   # v: no such column
    valid = (labels >= 0) & (labels < v)
    inv_n, z_w = torch.full((1,), 0.25, device=DEV), 1e-3
    stats, nll, lse2, worst = torch.zeros(2, device=DEV), 0.0, 0.0, 0.0
    got = logits.clone()
    cu.ce_fwd_bwd(got, labels, stats, inv_n, z_w, tiles)
    for lo in range(0, rows, 512):
        hi = min(rows, lo + 512)
        x, ok, at = logits[lo:hi].double(), valid[lo:hi], labels[lo:hi].clamp(0, v - 1)[:, None]
        lse = torch.logsumexp(x, -1, keepdim=True)
        nll, lse2 = nll + (lse - x.gather(1, at))[ok].sum(), lse2 + lse[ok].square().sum()
        terms = (x - lse).exp_().mul_(0.25 * (1 + 2 * z_w * lse)) * ok[:, None]
        want = terms.scatter_add(1, at, -0.25 * ok[:, None].double())
        # rounded to bf16 (2^-9); t - lse is right to 2^-24 * 256 and so is its exponential, before the label's one is taken off
        assert ((got[lo:hi].double() - want).abs() <= want.abs() * 2.0**-8 + terms * 2.0**-15 + 1e-30).all()
    assert torch.allclose(stats.double(), torch.stack([nll, lse2]), rtol=1e-5)
    again = logits.clone()   # the kernel that reads the rows itself
    sums = torch.zeros(2, device=DEV)
    cu.ce_fwd_bwd(again, labels, sums, inv_n, z_w)
    assert torch.allclose(stats, sums, rtol=1e-5) and native_lib.read_status() == 0


def test_products_of_other_kernels_leave_none(native_lib):
    for rows, v, k in [(8, 32000, 2048), (200, 1000, 2048), (2047, 1000, 2048), (2048, 32000, 2048), (2104, 32000, 1016)]:
        h, w = torch.randn(rows, k, device=DEV).bfloat16(), torch.randn(v, k, device=DEV).bfloat16()
        logits, tiles = native_lib.gemm_logits(h, w)
        assert tiles is None and torch.equal(logits, native_lib.gemm(h, w))


@pytest.mark.parametrize("rows,v,width", [(3840, 1032, 128), (512, 9480, 160), (1024, 6152, 192), (1152, 6152, 224), (2560, 4104, 192), (1001, 12000, 224)])
def test_tiles_of_every_width(native_lib, monkeypatch, rows, v, width):
    """The product takes narrower column tiles where 256 columns would leave the last round nearly empty."""
    assert native_lib.lib().kf_gemm_logits_width(rows, v, 64, native_lib.sm_count()) == width
    test_against_double(native_lib, monkeypatch, rows, v, 64)
