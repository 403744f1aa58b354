"""Projections over several weight matrices: how many there are and how they lie in memory.

The kernels read a matrix by its address and row pitch alone, so a weight they cannot describe has to be copied first.  On the
CPU the native entries are replaced by functions that read memory exactly as the kernels do."""

import ctypes

import pytest
import torch

DEV = "cuda"


def _read(ptr, rows, cols, pitch):
    """The (rows, cols) matrix the kernel sees: contiguous columns at a row pitch."""
    n = (rows - 1) * pitch + cols
    return torch.frombuffer((ctypes.c_int16 * n).from_address(ptr), dtype=torch.bfloat16).as_strided((rows, cols), (pitch, 1)).float()


class _FakeLibrary:
    def __init__(self):
        self.calls = []

    def _stack(self, ptrs, rows, cols, pitches):
        rows = list(rows) + [0]
        ws = list(zip(ptrs, rows, pitches))[: rows.index(0)]   # the first empty matrix ends the list
        if any(ld < cols or ld % 8 for _, _, ld in ws):   # a tensor map refuses these
            return None
        return torch.cat([_read(p, n, cols, ld) for p, n, ld in ws])

    def _store(self, out, y, ldo):
        m, n = y.shape
        buf = (ctypes.c_int16 * ((m - 1) * ldo + n)).from_address(out)
        torch.frombuffer(buf, dtype=torch.bfloat16).as_strided((m, n), (ldo, 1)).copy_(y.bfloat16())
        return 0

    def kf_gemm_skinny_bf16(self, x, w0, w1, w2, out, res, m, k, n0, n1, n2, ldx, l0, l1, l2, ldo, ldr, first, pdl, sms, st):
        self.calls.append("few rows")
        w = self._stack((w0, w1, w2), (n0, n1, n2), k, (l0, l1, l2))
        return 200 if w is None else self._store(out, _read(x, m, k, ldx) @ w.t(), ldo)

    def kf_gemm_rope_bf16(self, x, w0, w1, w2, out, m, n0, n1, n2, k, ldx, ldw, ldo, cos, sin, s, cols, hd, sms, st):
        self.calls.append("rope" if cols else "separate")
        assert not cols or (cos % 16 == 0 and sin % 16 == 0)   # read 16 bytes at a time
        w = self._stack((w0, w1, w2), (n0, n1, n2), k, (ldw,) * 3)
        return 200 if w is None else self._store(out, _read(x, m, k, ldx) @ w.t(), ldo)

    def kf_gemm_dgrad_stacked_bf16(self, dy, w0, w1, w2, out, m, k, n0, n1, n2, ldy, ldw, ldo, sms, st):
        self.calls.append("separate dgrad")
        w = self._stack((w0, w1, w2), (n0, n1, n2), k, (ldw,) * 3)
        return 200 if w is None else self._store(out, _read(dy, m, n0 + n1 + n2, ldy) @ w, ldo)

    def kf_gemm_k_pieces(self, m, n, k, sms):
        return 1

    def kf_gemm_bf16(self, a, b, out, res, m, n, k, lda, ldb, ldc, ldr, a_mn, b_mn, f32, acc, mode, sms, st):
        self.calls.append("tiles")
        am = _read(a, k, m, lda).t() if a_mn else _read(a, m, k, lda)
        bm = _read(b, k, n, ldb) if b_mn else _read(b, n, k, ldb).t()
        return self._store(out, am @ bm, ldc)

    def kf_rope_bf16(self, *a):
        self.calls.append("rotation")
        return 0


@pytest.fixture
def fake(monkeypatch):
    from kempnerforge_b200.ops import cuda as kc

    f = _FakeLibrary()
    monkeypatch.setattr(kc, "lib", lambda: f)
    monkeypatch.setattr(kc, "sm_count", lambda: 2)
    monkeypatch.setattr(kc, "_stream", lambda: 0)
    return f


def _weights(form, rows, k, device="cpu"):
    g = torch.Generator(device=device).manual_seed(3)
    out = []
    for n in rows:
        if form == "dense":
            w = torch.randn(n, k, device=device, generator=g).bfloat16()
        elif form == "columns":        # every second column: the row pitch alone says nothing about it
            w = torch.randn(n, 2 * k, device=device, generator=g).bfloat16()[:, ::2]
        elif form == "transposed":
            w = torch.randn(k, n, 8, device=device, generator=g).bfloat16()[..., 0].t()
        elif form == "one row":        # a row pitch of zero
            w = torch.randn(1, k, device=device, generator=g).bfloat16().expand(n, k)
        else:                          # rows cut out of a wider matrix
            w = torch.randn(n, k + 24, device=device, generator=g).bfloat16()[:, 8 : 8 + k]
        out.append(w)
    return out


def _bounded(got, p, q):
    """A bf16 rounding (2^-9) of an fp32 sum in any order."""
    want, mag = p.double() @ q.double(), p.double().abs() @ q.double().abs()
    return bool(((got.double() - want).abs() <= 2.0**-8 * want.abs() + 2.0**-16 * mag).all())


def _check(x, ws):
    from kempnerforge_b200.ops import functional as F

    xl = x.clone().requires_grad_(True)
    wl = [w.detach().requires_grad_(True) for w in ws]
    y = F._LinearFn.apply(xl, *wl)
    dy = torch.randn(y.shape, device=x.device, generator=torch.Generator(device=x.device).manual_seed(5)).bfloat16()
    got = torch.autograd.grad(y, [xl, *wl], dy)
    w = torch.cat([t.detach() for t in ws])
    assert y.shape == (x.shape[0], w.shape[0])
    assert _bounded(y.detach(), x, w.t())
    assert _bounded(got[0], dy, w)
    assert _bounded(torch.cat(got[1:]), dy.t(), x)


FORMS = ["dense", "columns", "transposed", "one row", "cut"]


@pytest.mark.parametrize("rows", [(16,) * 4, (8, 16, 24, 8, 8), (128, 64), (128, 128, 64), (128, 0, 64), (0, 64)])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("m", [3, 600])
def test_every_weight_counts_whatever_its_layout(fake, rows, form, m):
    _check(torch.randn(m, 64).bfloat16(), _weights(form, rows, 64))


def test_dense_weights_are_still_read_where_they_are(fake):
    _check(torch.randn(600, 64).bfloat16(), _weights("dense", (128, 64), 64))
    assert fake.calls[0] == "separate"
    fake.calls.clear()
    _check(torch.randn(3, 64).bfloat16(), _weights("cut", (128, 64), 64))
    assert fake.calls[0] == "few rows"


def test_more_than_three_matrices_are_refused_by_the_kernels_front_end(fake):
    from kempnerforge_b200.ops import cuda as kc

    with pytest.raises(AssertionError):
        kc.gemm_rows(torch.randn(3, 64).bfloat16(), _weights("dense", (16,) * 4, 64))


def test_a_matrix_on_another_device_is_refused_before_any_kernel(fake):
    from kempnerforge_b200.ops import cuda as kc

    x, w = torch.randn(3, 64).bfloat16(), _weights("dense", (128, 64), 64)
    for ws in ([w[0], w[1].to("meta")], [w[0].to("meta"), w[1].to("meta")]):
        with pytest.raises((AssertionError, RuntimeError, NotImplementedError)):
            kc.gemm_rows(x, ws)
        with pytest.raises((AssertionError, RuntimeError, NotImplementedError)):
            kc.dgrad_rows(torch.randn(600, 192).bfloat16(), ws)
    assert not fake.calls


@pytest.mark.parametrize("m", [8, 600])
def test_input_gradient_wants_rows_of_its_weights_width(fake, m):
    from kempnerforge_b200.ops import cuda as kc

    ws = _weights("dense", (128, 64), 64)
    for dy in (torch.randn(192, m).bfloat16().t(), torch.randn(m, 200).bfloat16(), torch.randn(m, 192).half()):
        with pytest.raises(AssertionError):
            kc.dgrad_rows(dy, ws)
    with pytest.raises((AssertionError, RuntimeError)):
        kc.dgrad_rows(torch.randn(m, 192).bfloat16(), [w.float() for w in ws])
    assert not fake.calls


def _tables(s, half, shift, device="cpu"):
    """cos | sin of one packed buffer that starts ``shift`` values late."""
    g = torch.Generator(device=device).manual_seed(2)
    ang = torch.rand(s, half, device=device, generator=g)
    buf = torch.empty(2 * s * half + shift, device=device)
    cos, sin = buf[shift : shift + s * half].view(s, half), buf[shift + s * half :].view(s, half)
    cos.copy_(ang.cos())
    sin.copy_(ang.sin())
    return cos, sin


@pytest.mark.parametrize("shift", [0, 1, 2, 4])
def test_rotary_tables_off_16_bytes_take_the_separate_rotation(fake, shift):
    from kempnerforge_b200.ops import cuda as kc
    from kempnerforge_b200.ops import fused_block

    x, ws = torch.randn(512, 64).bfloat16(), _weights("dense", (256, 128, 128), 64)
    cos, sin = _tables(256, 64, shift)
    kc.qkv_rope(x, ws, cos, sin, 256, 128)
    assert ("rope" in fake.calls) == (shift % 4 == 0) and ("rotation" in fake.calls) == (shift % 4 != 0)
    assert fused_block._rope_fused(x, torch.cat(ws), cos, sin, 256, 128) == (shift % 4 == 0)
    if shift % 4:
        with pytest.raises(AssertionError):
            kc.gemm(x, torch.cat(ws), rope=(cos, sin, 256, 384, 128))


@pytest.mark.gpu
@pytest.mark.parametrize("grad", [False, True])
def test_a_block_takes_rotary_tables_from_anywhere(native_lib, grad):
    from kempnerforge_b200.config import ModelConfig
    from kempnerforge_b200.models.transformer import TransformerBlock

    torch.manual_seed(0)
    block = TransformerBlock(ModelConfig(dim=512, n_layers=1, n_heads=4, n_kv_heads=2, vocab_size=256, ffn_hidden_dim=512,
                                         max_seq_len=512), 0).to(DEV, torch.bfloat16)
    x = torch.randn(2, 300, 512, device=DEV).bfloat16()
    out = []
    for shift in (0, 1):
        cos, sin = _tables(300, 64, shift, DEV)
        xl = x.clone().requires_grad_(grad)
        with torch.set_grad_enabled(grad):
            y = block(xl, cos, sin)
        out.append([y.detach()] + ([torch.autograd.grad(y.float().square().sum(), xl)[0]] if grad else []))
    assert native_lib.read_status() == 0
    for a, b in zip(*out):   # q, k and their gradients are rounded once more around the separate rotation (2^-9 each)
        assert float((a.float() - b.float()).norm()) <= 2.0**-6 * float(a.float().norm())


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [(64,) * 4, (128, 256, 64, 8, 512), (1024, 256, 256), (640, 640), (1024, 0, 512)])
@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("m", [5, 300, 4100])
def test_several_weights_on_the_gpu(native_lib, rows, form, m):
    x = torch.randn(m, 512, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1)).bfloat16()
    _check(x, _weights(form, rows, 512, DEV))
    assert native_lib.read_status() == 0
