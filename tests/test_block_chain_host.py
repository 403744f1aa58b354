"""Which addresses the native calls of a dense block are given (no GPU: the calls are recorded, not made)."""

import ctypes

import pytest
import torch
from torch.utils.checkpoint import checkpoint

from kempnerforge_b200.ops import fused_block

B, S, D, H, HD, F = 1, 320, 128, 2, 128, 256
N_OPERANDS = 12   # x, wn1, wq, wk, wv, wo, wn2, wg, wu, wd, cos, sin
N_PARTS = 10


class _Recorder:
    def __init__(self):
        self.calls = []

    def _note(self, which, ints):
        self.calls.append((which, list((ctypes.c_longlong * (N_OPERANDS + N_PARTS)).from_address(ints))))
        return 0

    def kf_block_train_fwd_bf16(self, ints, reals, stream):
        return self._note("fwd", ints)

    def kf_block_train_bwd_bf16(self, ints, reals, stream):
        return self._note("bwd", ints)

    def kf_rmsnorm_bwd_blocks(self, rows):
        return 1

    def of(self, which):
        return [c for w, c in self.calls if w == which]


@pytest.fixture
def calls(monkeypatch):
    rec = _Recorder()
    kc = fused_block.kc
    monkeypatch.setattr(kc, "lib", lambda: rec)
    monkeypatch.setattr(kc, "_stream", lambda: 0)
    monkeypatch.setattr(kc, "sm_count", lambda: 148)
    return rec


def _operands():
    shapes = ((D,), (H * HD, D), (H * HD, D), (H * HD, D), (D, H * HD), (D,), (F, D), (F, D), (D, F))
    weights = [torch.nn.Parameter(torch.randn(s).bfloat16()) for s in shapes]
    return weights, torch.randn(S, HD // 2), torch.randn(S, HD // 2)


def _block(x, weights, cos, sin):
    return fused_block.DenseBlockFn.apply(x, cos, sin, *weights, 1e-5, HD, False)


def test_backward_reads_the_tensors_that_autograd_hands_back(calls):
    weights, cos, sin = _operands()
    handed = []

    def unpack(t):
        handed.append(t)
        return t

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), unpack):
        x = torch.randn(B, S, D).bfloat16().requires_grad_(True)
        y = _block(x, weights, cos, sin)
    y.backward(torch.zeros_like(y))
    (fwd,), (bwd,) = calls.of("fwd"), calls.of("bwd")
    assert [bwd[0], bwd[10], bwd[11]] == [t.data_ptr() for t in handed] and not {bwd[0], bwd[10], bwd[11]} & {fwd[0], fwd[10], fwd[11]}
    assert bwd[1:10] == fwd[1:10] and bwd[N_OPERANDS:] == fwd[N_OPERANDS:]


def test_backward_inside_an_enclosing_checkpoint(calls):
    weights, cos, sin = _operands()
    x = torch.randn(B, S, D).bfloat16().requires_grad_(True)
    kept = []

    def body(t):
        t = t * 2
        kept.append(t)    # no address is used twice
        return _block(t, weights, cos, sin)

    y = checkpoint(body, x, use_reentrant=False)
    y.backward(torch.zeros_like(y))
    (first, again), (bwd,) = calls.of("fwd"), calls.of("bwd")
    assert bwd[0] == again[0] != first[0]


def test_backward_reads_a_weight_where_it_is_now(calls):
    weights, cos, sin = _operands()
    x = torch.randn(B, S, D).bfloat16().requires_grad_(True)
    y = _block(x, weights, cos, sin)
    old = [w.data for w in weights]   # their memory is not used again
    for w in weights:
        w.data = w.data.clone()
    y.backward(torch.zeros_like(y))
    (fwd,), (bwd,) = calls.of("fwd"), calls.of("bwd")
    assert bwd[1:10] == [w.data_ptr() for w in weights] and fwd[1:10] == [w.data_ptr() for w in old]
    assert not set(bwd[1:10]) & set(fwd[1:10])


def test_another_layout_in_the_backward(calls, monkeypatch):
    """A weight that the native call cannot read any more leaves the block to the op-by-op path; a strided input is copied."""
    weights, cos, sin = _operands()
    x = torch.randn(B, S, D).bfloat16().requires_grad_(True)
    wide = torch.empty(B * S, 2 * D, dtype=torch.bfloat16)

    def unpack(t):
        if t.shape != (B * S, D):
            return t
        wide[:, :D] = t
        return wide[:, :D]

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
        y = _block(x, weights, cos, sin)
    y.backward(torch.zeros_like(y))
    (bwd,) = calls.of("bwd")
    assert bwd[0] != wide.data_ptr()

    y = _block(x, weights, cos, sin)
    weights[2].data = torch.randn(D, H * HD).bfloat16().t()
    seen = []
    monkeypatch.setattr(fused_block, "_wgrad", lambda *a: seen.append(a) or (_ for _ in ()).throw(StopAsyncIteration))
    with pytest.raises(StopAsyncIteration):
        y.backward(torch.zeros_like(y))
    assert len(calls.of("bwd")) == 1 and len(seen) == 1
