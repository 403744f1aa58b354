"""The fp8 cast on ragged shapes and pitches: bytes must equal torch's conversion, nothing outside may be written."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e5m2", [False, True])
@pytest.mark.parametrize("rows,cols,pitch", [(16, 16, 16), (128, 128, 128), (129, 136, 136), (144, 272, 280), (2000, 4096, 4096),
                                            (1, 8, 8), (37, 131, 136), (15, 127, 127), (300, 520, 523)])
def test_cast_matches_torch_bytewise(native_lib, rows, cols, pitch, e5m2):
    g = torch.Generator(device="cuda").manual_seed(rows)
    base = (torch.randn(rows, pitch, device="cuda", generator=g) * 3).bfloat16()
    x = base[:, :cols]
    scale = native_lib.fp8_scale(x, e5m2)
    top, dt = (57344.0, torch.float8_e5m2) if e5m2 else (448.0, torch.float8_e4m3fn)
    assert torch.equal(scale, (torch.tensor(top, device="cuda") / x.float().abs().max()).reshape(1)) or \
        abs(float(scale) * float(x.float().abs().max()) / top - 1) < 2.0**-22   # one approximate division
    row, t = native_lib.fp8_cast(x, scale, e5m2, True, True)
    want = (x.float() * scale).clamp(-top, top).to(dt).view(torch.uint8)
    assert torch.equal(row, want) and torch.equal(t, want.t())
    only_t = native_lib.fp8_cast(x, scale, e5m2, False, True)
    assert only_t[0] is None and torch.equal(only_t[1], want.t())
    assert torch.equal(native_lib.fp8_cast(x, scale, e5m2, True, False)[0], want)


@pytest.mark.parametrize("rows", [16, 112, 128, 144, 2000])
def test_products_over_a_transposed_copy_do_not_see_its_padding(native_lib, rows):
    """The rows of the copy lie a multiple of 128 bytes apart; the bytes between them are not part of the product."""
    gen = torch.Generator(device="cuda").manual_seed(rows)
    a, b = (torch.randn(rows, n, device="cuda", generator=gen).bfloat16() for n in (272, 144))
    sa, sb = native_lib.fp8_scale(a, True), native_lib.fp8_scale(b)
    at, bt = native_lib.fp8_cast(a, sa, True, False, True)[1], native_lib.fp8_cast(b, sb, False, False, True)[1]
    assert at.shape == (272, rows) and at.stride(0) % 128 == 0 and bt.stride(0) % 128 == 0
    for t in (at, bt):   # 0x7f: NaN in both formats
        base = torch.as_strided(t, (t.shape[0], t.stride(0)), t.stride(), t.storage_offset())
        base[:, rows:] = 0x7F
    got = native_lib.gemm_fp8(at, bt, sa, sb, True, False)
    assert torch.equal(got, native_lib.gemm_fp8(at.contiguous(), bt.contiguous(), sa, sb, True, False))
    assert torch.isfinite(got).all() and native_lib.read_status() == 0
