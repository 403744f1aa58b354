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


def _parts(x, labels, z_w):
    """(sum of nll, sum of lse^2, gradient) of the rows with a label, in double."""
    x, ok = x.double(), labels >= 0
    lse = torch.logsumexp(x, -1)
    at = labels.clamp_min(0)[:, None]
    want = (x - lse[:, None]).exp() * (0.25 * (1 + 2 * z_w * lse))[:, None]
    return (lse - x.gather(1, at)[:, 0])[ok].sum(), lse[ok].square().sum(), (want.scatter_add(1, at, torch.full_like(at, -0.25, dtype=want.dtype)) * ok[:, None])


# Columns without a value: the words of one thread, the first and last ones, several tiles of columns, all but one
@pytest.mark.parametrize("masked", [[(0, 8)], [(8, 16)], [(0, 512), (1024, 2048)], [(4096, 4104)], [(0, 4103)], [(1, 4104)]])
@pytest.mark.parametrize("tiles", [True, False])
def test_masked_columns_add_nothing(native_lib, monkeypatch, tiles, masked):
    cu = native_lib
    monkeypatch.setattr(cu, "LOGITS_MIN_K", 0 if tiles else 1 << 30)
    monkeypatch.setattr(cu, "LOGITS_MIN_BYTES", 0)
    rows, v, k, z_w = 2560, 4104, 64, 1e-3
    torch.manual_seed(1)
    h, w = torch.randn(rows, k, device=DEV).bfloat16(), torch.randn(v, k, device=DEV).mul_(3 * k**-0.5).bfloat16()
    h[:, 0] = 1
    gone = torch.zeros(v, dtype=torch.bool, device=DEV)
    for a, b in masked:
        gone[a:b] = True
    w[gone, 0] = -torch.inf
    logits, stats_of_tiles = cu.gemm_logits(h, w)
    assert (stats_of_tiles is not None) == tiles and (logits[:, gone] == -torch.inf).all()
    labels = (~gone).nonzero()[:, 0][torch.randint(0, int((~gone).sum()), (rows,), device=DEV)]
    labels[::7] = -100
    nll, lse2, want = _parts(logits, labels, z_w)
    sums, inv_n = torch.zeros(2, device=DEV), torch.full((1,), 0.25, device=DEV)
    cu.ce_fwd_bwd(logits, labels, sums, inv_n, z_w, stats_of_tiles)
    assert (logits[:, gone] == 0).all()
    assert torch.allclose(sums.double(), torch.stack([nll, lse2]), rtol=1e-5, atol=1e-3)   # 2560 rows of fp32
    assert ((logits.double() - want).abs() <= want.abs() * 2.0**-8 + 0.25 * 2.0**-15).all()
    assert cu.read_status() == 0


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("tiles", [True, False])
def test_a_row_that_is_not_finite_is_reported_and_keeps_to_itself(native_lib, monkeypatch, tiles, bad):
    cu = native_lib
    monkeypatch.setattr(cu, "LOGITS_MIN_K", 0 if tiles else 1 << 30)
    monkeypatch.setattr(cu, "LOGITS_MIN_BYTES", 0)
    rows, v, k = 2560, 4104, 64
    torch.manual_seed(2)
    h, w = torch.randn(rows, k, device=DEV).bfloat16(), torch.randn(v, k, device=DEV).bfloat16()
    labels, inv_n = torch.randint(0, v, (rows,), device=DEV), torch.full((1,), 0.25, device=DEV)

    def call(h):
        logits, tiled = cu.gemm_logits(h, w)
        assert (tiled is not None) == tiles
        sums = torch.zeros(2, device=DEV)
        cu.ce_fwd_bwd(logits, labels, sums, inv_n, 0.0, tiled)
        return logits, sums

    clean, sums = call(h)
    assert torch.isfinite(sums).all() and torch.isfinite(clean).all()
    h[300, 5] = bad
    got, sums = call(h)
    others = torch.arange(rows, device=DEV) != 300
    assert not torch.isfinite(sums[0]) and got[300].isnan().any() and torch.equal(got[others], clean[others])


@pytest.mark.parametrize("v", [8, 4096, 4104, 4107])
def test_values_that_one_thread_alone_has_met(native_lib, v):
    """Eight words of -inf beside a NaN in the same thread's columns: the NaN stays one.  The vocabulary-parallel form alike."""
    logits = torch.zeros(4, v, device=DEV).bfloat16() if v % 8 == 0 else torch.zeros(4, -(-v // 8) * 8, device=DEV).bfloat16()[:, :v]
    logits[:, :8] = -torch.inf
    logits[1, 3] = torch.nan
    logits[2, v - 1] = torch.nan
    labels = torch.full((4,), v - 1, device=DEV)
    want = torch.logsumexp(logits.double(), -1)
    row_max, row_sum, _ = native_lib.ce_vp_stats(logits.clone() if v % 8 == 0 else logits, labels, 0)
    lse = torch.where(row_max == -torch.inf, 0, row_max) + row_sum.log()
    assert torch.allclose(lse.double(), want, rtol=1e-6, equal_nan=True)
    sums, inv_n = torch.zeros(2, device=DEV), torch.full((1,), 1.0, device=DEV)
    for r in (0, 1, 2, 3):
        row = torch.zeros(1, -(-v // 8) * 8, device=DEV).bfloat16()[:, :v].copy_(logits[r : r + 1])
        sums.zero_()
        native_lib.ce_fwd_bwd(row, labels[:1], sums, inv_n, 0.0)
        nll = want[r] - logits[r, v - 1].double()
        assert torch.allclose(sums[0].double(), nll, rtol=1e-6, atol=1e-6, equal_nan=True)
