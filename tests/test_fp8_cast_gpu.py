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
