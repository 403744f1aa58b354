"""FP8 training for dense Linear layers: tensorwise dynamic scaling, e4m3 activations / weights and e5m2
gradients, bf16 master weights, fp32 accumulation on tcgen05 ``kind::f8f6f4`` tensor cores.

``convert_model`` tags the weights of the selected ``nn.Linear`` modules; ``ops.functional.linear`` /
``fused_linear`` route tagged weights through ``_Fp8LinearFn``:

    forward   y  = (q4(x) @ q4(W)ᵀ)            / (s_x s_w)
    backward  dx = (q5(dy) @ q4(W))             / (s_g s_w)      q4 = e4m3, q5 = e5m2,
              dW = (q5(dy)ᵀ @ q4(x))            / (s_g s_x)      s = fp8_max / absmax (device scalars)

Scales never visit the host.  The cast kernel emits the transposed copies dgrad / wgrad need in the same pass,
so all three GEMMs run with the reduction dimension contiguous.  On a CPU (tests) the same arithmetic is
emulated with ``torch.float8_*`` dtypes.

Parity: kempnerforge/distributed/parallel.py:125-174 (torchao ``convert_to_float8_training`` with tensorwise
recipes; the module filter skips experts, shared experts and routers; dims must be multiples of 16).
"""

from __future__ import annotations

import torch
from torch import nn
from torch.multiprocessing.reductions import StorageWeakRef

from kempnerforge_b200.metrics.logger import get_logger

log = get_logger(__name__)

E4M3_MAX = 448.0
E5M2_MAX = 57344.0


def _eligible(linear: nn.Linear) -> bool:
    return linear.in_features % 16 == 0 and linear.out_features % 16 == 0


def convert_model(model: nn.Module, skip: tuple[str, ...] = ("experts", "shared_expert", "router")) -> int:
    """Tag every eligible ``nn.Linear`` outside ``skip`` for fp8 GEMMs.  Returns the number tagged."""
    n = 0
    for name, mod in model.named_modules():
        if not isinstance(mod, nn.Linear) or any(part in skip for part in name.split(".")):
            continue
        if name.split(".")[-1] == "proj" and "output_head" in name:
            continue  # the vocabulary projection stays bf16: it is fused with the loss
        if not _eligible(mod):
            continue
        mod.weight._kf_fp8 = True
        n += 1
    for m in model.modules():
        if hasattr(m, "ac_mode"):
            m._kf_fp8_block = True  # the fused bf16 block node is bypassed
    log.info("fp8: %d Linear layers use e4m3/e5m2 tensor-core GEMMs", n)
    return n


def is_fp8_weight(w: torch.Tensor) -> bool:
    return bool(getattr(w, "_kf_fp8", False))


# --------------------------------------------------------------------------- quantisation
def quantize(x2: torch.Tensor, e5m2: bool = False, want_row: bool = True, want_t: bool = False,
             scale=None):
    """(scale, row-major fp8 bytes or None, transposed fp8 bytes or None) of a 2-D bf16 tensor.  ``scale``: the one to use, or (on a GPU) the
    maxima that the kernel before took of ``x2``; else the largest magnitude is looked for."""
    from kempnerforge_b200.ops import cuda as cu

    if x2.is_cuda:
        if scale is None:
            scale = cu.fp8_absmax(x2)
        row, t = cu.fp8_cast(x2, scale, e5m2, want_row, want_t)
        return scale.scratch[:1] if isinstance(scale, cu.PartialMax) else scale, row, t
    fmax = E5M2_MAX if e5m2 else E4M3_MAX
    dt = torch.float8_e5m2 if e5m2 else torch.float8_e4m3fn
    if scale is None:
        scale = (fmax / x2.float().abs().max().clamp_min(1e-12)).reshape(1)
    q = (x2.float() * scale).clamp(-fmax, fmax).to(dt)
    return scale, (q if want_row else None), (q.t().contiguous() if want_t else None)


def scaled_mm(a8, b8, sa, sb, a_e5m2=False, b_e5m2=False, out=None, accumulate=False) -> torch.Tensor:
    """(a8 @ b8ᵀ) / (sa * sb) -> bf16; both operands (rows, K) with K contiguous."""
    from kempnerforge_b200.ops import cuda as cu

    if a8.is_cuda:
        return cu.gemm_fp8(a8, b8, sa, sb, a_e5m2, b_e5m2, out=out, accumulate=accumulate)
    y = (a8.float() @ b8.float().t()) / (sa * sb)
    if out is None:
        return y.to(torch.bfloat16)
    if accumulate:
        out.add_(y.to(out.dtype))
    else:
        out.copy_(y.to(out.dtype))
    return out


class _Copies:
    """The fp8 copies of (stacked) weights, kept on the first of them; a weight that is pickled or copied takes none along."""

    __slots__ = ("state", "storages", "scale", "row", "transposed")

    def __init__(self, state, storages, scale, row) -> None:
        self.state, self.storages, self.scale, self.row, self.transposed = state, storages, scale, row, None

    def __reduce__(self):
        return type(None), ()


def quantized_weight(weights, want_t: bool):
    """(scale, row-major fp8, transposed fp8 or None) of the weights stacked along the output dimension.

    The quantised copies are kept on the first weight tensor and reused until a weight is written, so the
    micro-batches, the recomputation and the backward pass of one step quantise each weight once instead of once per use.
    Tensor operations move a version counter; this package's optimizers and collectives, which write through raw pointers, move
    one or count their writes.  A program that writes a weight through ``.data`` or a pointer of its own,
    or replays a captured optimizer step, calls ``torch.autograd.graph.increment_version(weight)`` after it.
    Copies are reused on the stream that made them only, and neither taken into a captured graph nor out of it: a replay
    reads the weights as they are then."""
    from kempnerforge_b200.ops import functional as F

    stacked = lambda: F._stack_weight_rows(weights).detach()  # noqa: E731
    state = [0]
    if weights[0].is_cuda:
        if torch._C._cuda_isCurrentStreamCapturing():
            return quantize(stacked(), want_t=want_t)
        state[0] = torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())
    for w in weights:
        # its version, its address, the writes of kernels, and the version of the flat buffer that it is a view of (binding a
        # parameter to the buffer leaves it a counter of its own, which a write of the buffer does not move)
        own = w.__dict__.get
        flat = own("_kf_flat")
        state += w._version, w.data_ptr(), own("_kf_writes"), None if flat is None else flat.values_version
    holder = weights[0]
    cached = getattr(holder, "_kf_fp8_cache", None)
    # where the storage that held an address is alive, no other one does
    if type(cached) is not _Copies or cached.state != state or any([torch.UntypedStorage._expired(ref.cdata) for ref in cached.storages]):
        sw, w8, _ = quantize(stacked())
        cached = holder._kf_fp8_cache = _Copies(state, [StorageWeakRef(w.untyped_storage()) for w in weights], sw, w8)
    if want_t and cached.transposed is None:
        cached.transposed = quantize(stacked(), want_row=False, want_t=True, scale=cached.scale)[2]
    return cached.scale, cached.row, cached.transposed


class _Fp8LinearFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, *weights):
        x2 = x.reshape(-1, x.shape[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        sx, x8, _ = quantize(x2)
        sw, w8, _ = quantized_weight(weights, want_t=False)
        y = scaled_mm(x8, w8, sx, sw)
        ctx.save_for_backward(x2, sx, *weights)
        ctx.x_shape = x.shape
        return y.view(*x.shape[:-1], w8.shape[0])

    @staticmethod
    def backward(ctx, dy):
        from kempnerforge_b200.ops import functional as F

        x2, sx, *weights = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        need_dx = ctx.needs_input_grad[0]
        need_dw = any(ctx.needs_input_grad[1:])
        sg, g8, g8t = quantize(dy2, e5m2=True, want_row=need_dx, want_t=need_dw)
        dx = None
        if need_dx:
            sw, _, w8t = quantized_weight(weights, want_t=True)                     # (K, N)
            dx = scaled_mm(g8, w8t, sg, sw, a_e5m2=True).view(ctx.x_shape)
        wgrads = [None] * len(weights)
        if need_dw:
            _, _, x8t = quantize(x2, want_row=False, want_t=True, scale=sx)          # (K, T)
            wgrads = F._deposit_stacked_weight_grads(
                weights, ctx.needs_input_grad[1:],
                lambda out, acc: scaled_mm(g8t, x8t, sg, sx, a_e5m2=True, out=out, accumulate=acc))
        return (dx, *wgrads)


class _Fp8SwiGLUFn(torch.autograd.Function):
    """down(silu(x Wgᵀ) * (x Wuᵀ)) with fp8 products as one node: the arithmetic of two :class:`_Fp8LinearFn` around the SwiGLU
    kernel, except that the SwiGLU and its gradient, and the maxima that the casts of their results wait for, are taken in the
    epilogues of the products before them.  The hidden activation is cast once: where a gradient of ``wd`` will be wanted
    (``recording``) its transposed fp8 copy is written together with the other one and kept in its stead, at half its bytes.  The
    pre-activations are written only where they will be read, too."""

    @staticmethod
    def forward(ctx, x, wg, wu, wd, recording):
        from kempnerforge_b200.ops import cuda as cu

        x2 = x.reshape(-1, x.shape[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        sx, x8, _ = quantize(x2)
        s_gu, w8, _ = quantized_weight((wg, wu), want_t=False)
        gu, h, h_max = cu.gemm_fp8_swiglu(x8, w8, sx, s_gu, want_gu=recording and any(ctx.needs_input_grad[:3]))
        sh, h8, h8t = quantize(h, scale=h_max, want_t=recording and ctx.needs_input_grad[3])
        sd, d8, _ = quantized_weight((wd,), want_t=False)
        y = scaled_mm(h8, d8, sh, sd)
        ctx.save_for_backward(x2, sx, gu, h8t, sh, wg, wu, wd)
        ctx.x_shape = x.shape
        return y.view(*x.shape[:-1], d8.shape[0])

    @staticmethod
    def backward(ctx, dy):
        from kempnerforge_b200.ops import cuda as cu
        from kempnerforge_b200.ops import functional as F

        x2, sx, gu, h8t, sh, wg, wu, wd = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        need_x, need_g, need_u, need_d, _ = ctx.needs_input_grad
        need_h = need_x or need_g or need_u
        sg, g8, g8t = quantize(dy2, e5m2=True, want_row=need_h, want_t=need_d)
        dx = g_wg = g_wu = g_wd = None
        if need_h:
            sd, _, d8t = quantized_weight((wd,), want_t=True)
            dgu, dgu_max = cu.gemm_fp8_swiglu_bwd(g8, d8t, sg, sd, gu)
        if need_d:
            (g_wd,) = F._deposit_stacked_weight_grads(
                [wd], (True,), lambda out, acc: scaled_mm(g8t, h8t, sg, sh, a_e5m2=True, out=out, accumulate=acc))
        if need_h:
            need_w = need_g or need_u
            s_dgu, q8, q8t = quantize(dgu, e5m2=True, want_row=need_x, want_t=need_w, scale=dgu_max)
            if need_x:
                s_gu, _, w8t = quantized_weight((wg, wu), want_t=True)
                dx = scaled_mm(q8, w8t, s_dgu, s_gu, a_e5m2=True).view(ctx.x_shape)
            if need_w:
                _, _, x8t = quantize(x2, want_row=False, want_t=True, scale=sx)
                g_wg, g_wu = F._deposit_stacked_weight_grads(
                    [wg, wu], (need_g, need_u),
                    lambda out, acc: scaled_mm(q8t, x8t, s_dgu, sx, a_e5m2=True, out=out, accumulate=acc))
        return dx, g_wg, g_wu, g_wd, None


def swiglu_mlp(x: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor, wd: torch.Tensor) -> torch.Tensor | None:
    """A SwiGLU feed-forward whose three weights are tagged for fp8 and that the node covers, else None."""
    from kempnerforge_b200.ops import functional as F

    if (not F.use_native(x) or x.numel() == 0 or not supported(x, [wg, wu, wd]) or wg.shape != wu.shape
            or wd.shape[1] != wg.shape[0] or wg.shape[1] != x.shape[-1] or any(not w.is_cuda or w.dtype != torch.bfloat16 for w in (wg, wu, wd))):
        return None
    return _Fp8SwiGLUFn.apply(x, wg, wu, wd, torch.is_grad_enabled())


def linear(x: torch.Tensor, weights: list[torch.Tensor]) -> torch.Tensor:
    """fp8 Linear against one weight or several weights stacked along the output dimension."""
    return _Fp8LinearFn.apply(x, *weights)


def supported(x: torch.Tensor, weights: list[torch.Tensor]) -> bool:
    t = x.numel() // x.shape[-1]
    return (x.dtype == torch.bfloat16 and t % 16 == 0 and all(is_fp8_weight(w) for w in weights)
            and all(w.shape[0] % 16 == 0 and w.shape[1] % 16 == 0 for w in weights))
