"""ctypes binding of ``libkfb200.so`` — the hand-written sm_100a kernels.

Tensors are passed as raw device pointers together with the current CUDA
stream, so every launch is ordered like an ordinary PyTorch op.  Importing this
module on a machine with a GPU but without the built library raises: there is
no silent fallback to library kernels.
"""

from __future__ import annotations

import ctypes
import importlib.util
import math
import os
from array import array
from ctypes import c_float, c_int, c_longlong, c_void_p
from typing import NamedTuple

import torch

from kempnerforge_b200.metrics.logger import get_logger
from kempnerforge_b200.ops.build import LIB_PATH, STEPS_PATH

_lib = None
GEMM_MODE = int(os.environ.get("KF_GEMM_MODE", "0"))  # 0 = automatic, 1 = single CTA tiles, 2 = CTA pairs
LAUNCH_COUNT = 0  # number of native kernel launches issued through this module (bench bookkeeping)


class NativeKernelError(RuntimeError):
    pass


def lib() -> ctypes.CDLL:
    global _lib
    if _lib is None:
        if not LIB_PATH.exists():
            raise NativeKernelError(
                f"native library {LIB_PATH} is missing; run `python -m kempnerforge_b200.ops.build`"
            )
        _lib = ctypes.CDLL(str(LIB_PATH))
        _declare(_lib)
        if os.environ.get("KF_ATTN_BWD_DQ", "") == "red" and hasattr(_lib, "kf_attn_bwd_dq_mode"):
            _lib.kf_attn_bwd_dq_mode(0)
        if os.environ.get("KF_GROUPED_PAIR", "1") == "0" and hasattr(_lib, "kf_grouped_pair_mode"):
            _lib.kf_grouped_pair_mode(0)
    return _lib


def available() -> bool:
    return torch.cuda.is_available() and LIB_PATH.exists()


def _declare(L: ctypes.CDLL) -> None:
    vp, i, ll, f = c_void_p, c_int, c_longlong, c_float
    sigs = {
        "kf_gemm_k_pieces": [i, i, i, i],
        "kf_gemm_tokens_width": [i, i, i, i, i, i],
        "kf_gemm_split_k_bf16": [vp, vp, vp, vp, i, i, i, i, i, i, i, i, vp],
        "kf_gemm_bf16": [vp, vp, vp, vp, i, i, i, i, i, i, i, i, i, i, i, i, i, vp],
        "kf_gemm_swiglu_bf16": [vp, vp, vp, vp, vp, i, i, i, i, i, i, i, i, vp],
        "kf_gemm_rope_bf16": [vp, vp, vp, vp, vp, i, i, i, i, i, i, i, i, vp, vp, i, i, i, i, vp],
        "kf_gemm_dgrad_stacked_bf16": [vp, vp, vp, vp, vp, i, i, i, i, i, i, i, i, i, vp],
        "kf_gemm_skinny_bf16": [vp] * 6 + [i] * 14 + [vp],
        "kf_gemm_skinny_swiglu_bf16": [vp] * 4 + [i] * 9 + [vp],
        "kf_skinny_norm_rows": [],
        "kf_gemm_skinny_norm_swiglu_bf16": [vp, vp, f, vp, vp, vp] + [i] * 9 + [vp],
        "kf_gemm_skinny_norm_qkv_bf16": [vp, vp, f] + [vp] * 6 + [i] * 11 + [ll, vp, vp, i, i, vp],
        "kf_attn_fwd_pdl_bf16": [vp] * 6 + [i] * 6 + [ll] * 4 + [f, i, i, vp],
        "kf_rmsnorm_fwd_pdl_bf16": [vp, vp, vp, vp, i, i, f, i, vp],
        "kf_attn_decode_bf16": [vp] * 4 + [i] * 5 + [ll] * 5 + [f, i, i, i, vp],
        "kf_block_decode_bf16": [vp, vp, vp],
        "kf_blocks_decode_bf16": [vp, vp, i, vp],
        "kf_block_train_fwd_bf16": [vp, vp, vp],
        "kf_block_train_bwd_bf16": [vp, vp, vp],
        "kf_gemm_swiglu_bwd_bf16": [vp, vp, vp, vp, i, i, i, i, i, i, i, vp],
        "kf_gemm_symm_bf16": [i, vp, vp, vp, i, i, i, i, i, f, f, f, i, vp],
        "kf_rmsnorm_fwd_bf16": [vp, vp, vp, vp, i, i, f, vp],
        "kf_rmsnorm_bwd_blocks": [i],
        "kf_rmsnorm_bwd_bf16": [vp, vp, vp, vp, vp, vp, vp, vp, i, i, vp, vp],
        "kf_rope_bf16": [vp, vp, vp, vp, ll, i, i, i, i, i, vp],
        "kf_swiglu_fwd_bf16": [vp, vp, ll, i, vp],
        "kf_swiglu_bwd_bf16": [vp, vp, vp, ll, i, vp],
        "kf_embedding_fwd_bf16": [vp, vp, vp, ll, i, i, vp],
        "kf_embedding_bwd_bf16": [vp, vp, vp, ll, i, i, vp],
        "kf_ce_fwd_bwd_bf16": [vp, vp, vp, vp, vp, f, i, i, i, vp],
        "kf_cache_rows_bf16": [vp, ll, vp, vp, i, i, i, ll, vp],
        "kf_ce_grad_bf16": [vp, vp, i, vp, vp, vp, vp, vp, f, i, i, i, vp],
        "kf_gemm_logits_width": [i, i, i, i],
        "kf_gemm_logits_bf16": [vp, vp, vp, vp, i, i, i, i, i, i, i, vp],
        "kf_scale_bf16": [vp, ll, vp, vp],
        "kf_ce_vp_stats_bf16": [vp, vp, ll, vp, vp, vp, i, i, i, vp],
        "kf_ce_vp_bwd_bf16": [vp, vp, ll, vp, vp, vp, f, i, i, i, vp],
        "kf_adamw_flat": [vp, vp, vp, vp, ll, ll, f, f, f, f, f, f, f, vp, vp, i, i, i, vp],
        "kf_sumsq": [vp, ll, i, vp, vp, i, vp],
        "kf_test_flag_timeout": [vp, i, ll],
        "kf_gemm_fp8": [vp, vp, vp, i, i, i, ll, ll, i, i, i, vp, vp, i, i, vp],
        "kf_fp8_scale_bf16": [vp, ll, i, vp, vp, vp],
        "kf_gemm_fp8_swiglu": [vp, vp, vp, vp, i, i, i, ll, ll, i, i, vp, vp, vp, vp, i, vp],
        "kf_gemm_fp8_swiglu_bwd": [vp, vp, vp, vp, i, i, i, ll, ll, i, vp, vp, vp, vp, i, vp],
        "kf_fp8_absmax_bf16": [vp, ll, vp, vp, vp],
        "kf_fp8_cast_bf16": [vp, i, i, ll, vp, i, vp, i, vp, ll, vp, ll, vp],
        "kf_lion": [vp, vp, vp, ll, i, f, f, f, f, vp],
        "kf_sf_adamw": [vp, vp, vp, vp, vp, ll, i, f, f, f, f, f, f, f, i, vp],
        "kf_ep_put_bf16": [vp, vp, i, vp, i, i, i, i, ll, vp, vp, i, vp],
        "kf_ep_layout": [vp, i, i, vp, vp, vp, vp, vp],
        "kf_ep_move_bf16": [vp, vp, vp, vp, vp, i, i, i, ll, i, vp, vp],
        "kf_router_topk": [vp, i, vp, i, i, i, i, i] + [vp] * 10,
        "kf_router_bwd": [vp, i, vp, i, vp, vp, vp, i, vp, vp, vp, vp, i, i, i, vp, vp, i, vp, vp],
        "kf_grouped_experts_bf16": [i, vp, vp, vp, i, vp, vp, vp, i, i, i, i, ll, ll, ll, i, i, vp],
        "kf_moe_sort": [vp, i, i, vp, vp, vp, vp, vp],
        "kf_moe_capacity_mask": [vp, i, i, i, i, vp, vp],
        "kf_moe_gather_bf16": [vp, vp, i, i, i, vp, vp],
        "kf_moe_combine_bf16": [vp, vp, vp, i, vp, i, i, i, vp, vp],
        "kf_moe_combine_bwd_bf16": [vp, vp, vp, vp, i, i, i, i, vp, vp, vp],
        "kf_grouped_gemm_bf16": [vp, vp, vp, vp, i, i, i, i, ll, ll, i, i, vp],
        "kf_grouped_gemm_acc_bf16": [vp, vp, vp, vp, i, i, i, i, ll, ll, i, i, i, vp],
        "kf_grouped_swiglu_bf16": [vp, vp, vp, vp, vp, vp, i, i, i, i, ll, ll, ll, i, i, vp],
        "kf_grouped_swiglu_bwd_bf16": [vp, vp, vp, vp, vp, i, i, i, i, ll, ll, i, i, vp],
        "kf_swiglu_bwd_ragged_bf16": [vp, vp, vp, ll, vp, i, vp],
        "kf_grouped_wgrad_bf16": [vp, vp, vp, vp, i, i, i, i, ll, ll, i, vp],
        "kf_ag_gemm_bf16": [vp, vp, vp, vp, vp, i, i, i, i, ll, ll, ll, i, i, i, i, i, vp],
        "kf_gemm_rs_bf16": [vp, vp, vp, vp, vp, vp, i, i, i, i, ll, ll, i, i, i, i, i, vp],
        "kf_attn_bwd_bf16": [vp] * 12 + [i] * 6 + [ll] * 8 + [f, i, vp],
        "kf_attn_bwd_rope_bf16": [vp] * 12 + [i] * 6 + [ll] * 8 + [f, i, vp, vp, vp, vp],
        "kf_doc_blocks": [vp, i, vp, vp, i, i, vp],
        "kf_attn_bwd_dq_mode": [i],
        "kf_grouped_pair_mode": [i],
        "kf_attn_fwd2_bf16": [vp] * 7 + [i] * 6 + [ll] * 4 + [f, i, vp],
        "kf_attn_fwd_bf16": [vp, vp, vp, vp, vp, vp, i, i, i, i, i, i, ll, ll, ll, ll, f, i, vp],
        "kf_symm_rs_norm_bf16": [vp, vp, i, i, ll, ll, vp, vp, i, i, vp],
        "kf_symm_adamw_bcast_bf16": [vp, vp, i, i, vp, vp, vp, ll, ll, ll, f, f, f, f, f, f, f, vp, vp, i, vp],
        "kf_symm_gather_bf16": [vp, vp, i, i, ll, ll, i, vp],
        "kf_symm_pull_bf16": [vp, i, i, vp, vp, vp, vp, i, vp],
        "kf_symm_rs_shard_bf16": [vp, vp, i, i, i, vp, vp, vp, vp, i, i, vp],
        "kf_gemm_gather_bf16": [i, vp, vp, vp, i, i, i, i, i, i, vp, i, i, i, vp, vp, vp, vp, vp, vp, i, i, i, i, vp],
        "kf_read_status": [],
        "kf_clear_status": [],
        "kf_status_device_ptr": [],
    }
    for name, args in sigs.items():
        fn = getattr(L, name, None)
        if fn is None:
            continue
        fn.argtypes = args
        fn.restype = c_void_p if name == "kf_status_device_ptr" else c_int
    if hasattr(L, "kf_clear_status"):
        L.kf_clear_status.restype = None


def _stream() -> int:
    # the raw handle of the current stream of the current device, without building a Stream object around it
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _check(code: int, what: str, launches: int = 1) -> None:
    global LAUNCH_COUNT
    LAUNCH_COUNT += launches
    if code != 0:
        raise NativeKernelError(f"{what} failed with code {code}")


_SM_COUNT: dict[int, int] = {}


def sm_count() -> int:
    n = _SM_COUNT.get(torch._C._cuda_getDevice())
    if n is None:
        dev = torch.cuda.current_device()
        n = _SM_COUNT[dev] = torch.cuda.get_device_properties(dev).multi_processor_count
    return n


def read_status() -> int:
    """Status word of the library on the current device (0 = no kernel gave up a wait). Synchronises."""
    return int(lib().kf_read_status())


def clear_status() -> None:
    lib().kf_clear_status()


# --------------------------------------------------------------------------- row stacking of adjacent views
def rows_adjacent(tensors) -> bool:
    """True when 2-D tensors with equal width sit back to back in one storage (so they form one matrix)."""
    first = tensors[0]
    if first is None or not first.is_contiguous():
        return False
    ptr = first.data_ptr() + first.numel() * first.element_size()
    for t in tensors[1:]:
        if (
            t is None
            or not t.is_contiguous()
            or t.shape[1:] != first.shape[1:]
            or t.dtype != first.dtype
            or t.data_ptr() != ptr
            or t.untyped_storage().data_ptr() != first.untyped_storage().data_ptr()
        ):
            return False
        ptr += t.numel() * t.element_size()
    return True


def stack_rows(tensors):
    """One (sum rows, cols) matrix over the given row blocks: a zero-copy view when adjacent, else a copy."""
    tensors = list(tensors)
    if len(tensors) == 1:
        return tensors[0]
    if rows_adjacent(tensors):
        first = tensors[0]
        rows = sum(t.shape[0] for t in tensors)
        return torch.as_strided(first.detach(), (rows, *first.shape[1:]), first.stride())
    return torch.cat([t.detach() for t in tensors], dim=0)


# --------------------------------------------------------------------------- GEMM
# From this reduction length on (the input gradient of a vocabulary projection) the native rule for a split along K is asked; it
# never splits into pieces shorter than half of it.
SPLIT_K_MIN = 8192


def gemm(
    a: torch.Tensor,
    b: torch.Tensor,
    a_kmajor: bool = True,
    b_kmajor: bool = True,
    out: torch.Tensor | None = None,
    accumulate: bool = False,
    out_dtype: torch.dtype | None = None,
    residual: torch.Tensor | None = None,
    mode: int | None = None,
    rope: tuple | None = None,
) -> torch.Tensor:
    """out[M,N] = A * Bᵀ (+ out if ``accumulate``) (+ ``residual``) on the tcgen05 tensor cores.

    ``rope = (cos, sin, seq_len, rope_cols, head_dim)``: rotary position embedding in the epilogue (fused Q | K | V
    projection): the heads inside the first ``rope_cols`` output columns are rotated by the angle of position
    ``row % seq_len``; ``cos`` / ``sin`` are fp32 (seq_len, head_dim / 2).  Needs K-major operands, bf16 output.

    ``mode``: None/0 = automatic, 1 = single-CTA 128x256 tiles, 2 = CTA pairs (cta_group::2) on 256x256 tiles, 3 = CTA pairs
    on tiles cut to the number of rows.

    ``a_kmajor``: a is stored (M, K); otherwise (K, M).  ``b_kmajor``: b is stored (N, K); otherwise (K, N).
    Rows may be strided (row pitch a multiple of 8 elements); columns must be contiguous.
    """
    assert a.dtype == torch.bfloat16 and b.dtype == torch.bfloat16
    assert a.dim() == 2 and b.dim() == 2 and a.stride(1) == 1 and b.stride(1) == 1
    M, K = (a.shape[0], a.shape[1]) if a_kmajor else (a.shape[1], a.shape[0])
    N, Kb = (b.shape[0], b.shape[1]) if b_kmajor else (b.shape[1], b.shape[0])
    assert K == Kb, f"inner dimensions differ: {K} vs {Kb}"
    assert a.device == b.device, f"operands on {a.device} and {b.device}"
    lda, ldb = a.stride(0), b.stride(0)
    if out is None:
        out = torch.empty((M, N), dtype=out_dtype or torch.bfloat16, device=a.device)
        accumulate = False
    assert out.shape == (M, N) and out.stride(1) == 1
    ldc = out.stride(0)
    out_f32 = out.dtype == torch.float32
    assert out_f32 or out.dtype == torch.bfloat16
    if lda % 8 or ldb % 8 or ldc % (4 if out_f32 else 8) or a.data_ptr() % 16 or b.data_ptr() % 16 or out.data_ptr() % 16:
        raise NativeKernelError(
            f"gemm operands must have 16-byte aligned bases and row pitches (lda={lda}, ldb={ldb}, ldc={ldc})"
        )
    if rope is not None:
        assert a_kmajor and b_kmajor and not accumulate and residual is None
        return _gemm_rope(a, [b], out, rope)
    if (mode in (None, 0) and GEMM_MODE == 0 and _few_rows(M, N) and a_kmajor and b_kmajor and not out_f32
            and not accumulate and N % 8 == 0 and K % 8 == 0):
        return _stream_rows(a, [b], residual, out)
    ldr = 0
    if residual is not None:
        assert residual.shape == (M, N) and residual.dtype == out.dtype and residual.stride(1) == 1
        ldr = residual.stride(0)
        if ldr % (4 if out_f32 else 8) or residual.data_ptr() % 16:
            raise NativeKernelError("gemm residual must be 16-byte aligned")
    if (K >= SPLIT_K_MIN and mode in (None, 0) and GEMM_MODE == 0 and a_kmajor and not b_kmajor and not out_f32 and not accumulate
            and residual is None):
        pieces = lib().kf_gemm_k_pieces(M, N, K, sm_count())
        if pieces > 1:
            ws = torch.empty((pieces, M, N), dtype=torch.float32, device=a.device)
            _check(lib().kf_gemm_split_k_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), ws.data_ptr(), M, N, K, lda, ldb, ldc, pieces,
                                              sm_count(), _stream()), "kf_gemm_split_k_bf16", 2)
            return out
    code = lib().kf_gemm_bf16(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), residual.data_ptr() if residual is not None else None,
        M, N, K, lda, ldb, ldc, ldr, 0 if a_kmajor else 1, 0 if b_kmajor else 1, int(out_f32), int(accumulate),
        GEMM_MODE if mode is None else mode, sm_count(), _stream(),
    )
    _check(code, "kf_gemm_bf16")
    return out


# --------------------------------------------------------------------------- few rows / separate weights
# Up to this many rows of x the weight-streaming kernel (csrc/gemm_skinny_tcgen05.cu) is considered at all.
SKINNY_MAX_ROWS = 256


def _few_rows(m: int, n: int) -> bool:
    """Whether the weight-streaming kernel beats the 128 x 256 tiles for (m, n): always up to 64 rows (equal at worst, where
    the tiles fill the machine by themselves), above while the tiles leave half of the SMs idle.  Measured, L2 flushed, us
    (streaming / tiles): 1 x 4096, K 4096: 18 / 33; 64 x 28672, K 4096: 58 / 58; 128 x 28672: 71 / 59 (112 tiles);
    256 x 6144: 32 / 39 (48 tiles); 256 x 4096, K 14336: 51 / 98 (32 tiles); 128 x 32000, K 768: 29 / 23 (125 tiles)."""
    return m <= 64 or (m <= SKINNY_MAX_ROWS and 2 * (-(-n // 256)) * (-(-m // 128)) <= sm_count())


def _ptr(t: torch.Tensor | None):
    return t.data_ptr() if t is not None else None


def _plain_rows(w: torch.Tensor, device: torch.device) -> bool:
    """A kernel can read the matrix by its address and row pitch: on its GPU, not empty (an empty one ends the kernels' list),
    adjacent columns, rows that do not overlap, 16-byte steps.  Anything else is left to the copy that stacks the matrices: the pitch alone would name other elements, the address
    other memory."""
    return (w.device == device and w.shape[0] > 0 and w.stride(1) == 1 and w.stride(0) >= w.shape[1] and w.stride(0) % 8 == 0
            and w.data_ptr() % 16 == 0)


def _weights3(weights):
    """(pointers, rows, row pitches) of up to three stacked matrices, padded with empty ones."""
    n = 3 - len(weights)
    return ([w.data_ptr() for w in weights] + [None] * n, [w.shape[0] for w in weights] + [0] * n,
            [w.stride(0) for w in weights] + [0] * n)


def gemm_rows(x2: torch.Tensor, weights, residual: torch.Tensor | None = None, out: torch.Tensor | None = None) -> torch.Tensor:
    """x2 (M, K) times up to three (n_i, K) weights stacked along the output (+ ``residual``) -> bf16 (M, sum n_i).  With few
    rows the weights are read where they are; otherwise they are stacked for the tile kernels."""
    assert 1 <= len(weights) <= 3, "more than three matrices have to be stacked first"
    m, k = x2.shape
    if len(weights) > 1 and residual is None and out is None and _separate_ok(x2, weights, 128) and not rows_adjacent(weights):
        # the rotary kernel with nothing to rotate: one tensor map per weight
        n = sum(w.shape[0] for w in weights)
        out = torch.empty((m, n), dtype=torch.bfloat16, device=x2.device)
        ptrs, rows, pitch = _weights3(weights)
        _check(lib().kf_gemm_rope_bf16(x2.data_ptr(), *ptrs, out.data_ptr(), m, *rows, k, x2.stride(0), pitch[0], n, None, None,
                                       1, 0, 64, sm_count(), _stream()), "kf_gemm_rope_bf16")
        return out
    if not _few_rows(m, sum(w.shape[0] for w in weights)) or any(w.shape[0] % 8 or not _plain_rows(w, x2.device) for w in weights) or k % 8:
        return gemm(x2, stack_rows(weights), residual=residual, out=out)
    return _stream_rows(x2, weights, residual, out)


def _stream_rows(x2: torch.Tensor, weights, residual: torch.Tensor | None, out: torch.Tensor | None) -> torch.Tensor:
    """:func:`gemm_rows` on the weight-streaming kernel."""
    m, k = x2.shape
    ptrs, rows, pitch = _weights3(weights)
    n = sum(rows)
    if out is None:
        out = torch.empty((m, n), dtype=torch.bfloat16, device=x2.device)
    ldr = 0
    if residual is not None:
        assert residual.shape == (m, n) and residual.dtype == torch.bfloat16 and residual.stride(1) == 1
        ldr = residual.stride(0)
        if ldr % 8 or residual.data_ptr() % 16:
            raise NativeKernelError("gemm residual must be 16-byte aligned")
    if x2.stride(0) % 8 or x2.data_ptr() % 16 or out.stride(0) % 8 or out.data_ptr() % 16:
        raise NativeKernelError("gemm operands must have 16-byte aligned bases and row pitches")
    _check(lib().kf_gemm_skinny_bf16(x2.data_ptr(), *ptrs, out.data_ptr(), residual.data_ptr() if residual is not None else None,
                                     m, k, *rows, x2.stride(0), *pitch, out.stride(0), ldr, 0, 0, sm_count(), _stream()),
           "kf_gemm_skinny_bf16")
    return out


def _separate_ok(x2: torch.Tensor, weights, step: int) -> bool:
    """The CTA-pair kernel may read the weights through a tensor map each: enough 256 x 256 tiles for it, one pitch, all but
    the last matrix a multiple of ``step`` rows, heads of 64 columns throughout."""
    m, n = x2.shape[0], sum(w.shape[0] for w in weights)
    tiles = -(-m // 256) * (-(-n // 256))
    return (tiles >= 2 * (sm_count() // 2) and n % 64 == 0 and x2.stride(0) % 8 == 0 and x2.data_ptr() % 16 == 0
            and all(w.shape[0] % step == 0 for w in weights[:-1])
            and all(w.stride() == weights[0].stride() and _plain_rows(w, x2.device) for w in weights))


def dgrad_rows(dy2: torch.Tensor, weights) -> torch.Tensor:
    """dy2 (M, sum n_i) times the (n_i, K) weights stacked along n: the input gradient of :func:`gemm_rows`."""
    m, n = dy2.shape
    k = weights[0].shape[1]
    if (len(weights) in (2, 3) and not rows_adjacent(weights) and m > 0 and k > 0 and k % 8 == 0 and GEMM_MODE == 0
            and (n < SPLIT_K_MIN or lib().kf_gemm_k_pieces(m, k, n, sm_count()) == 1)
            and dy2.dtype == torch.bfloat16 and dy2.stride(1) == 1 and dy2.stride(0) % 8 == 0 and dy2.data_ptr() % 16 == 0
            and n == sum(w.shape[0] for w in weights) and all(w.shape[0] % 64 == 0 for w in weights[:-1])
            and all(w.dtype == torch.bfloat16 and w.shape[1] == k and w.stride() == weights[0].stride() and _plain_rows(w, dy2.device)
                    for w in weights)):
        out = torch.empty((m, k), dtype=torch.bfloat16, device=dy2.device)
        ptrs, rows, pitch = _weights3(weights)
        _check(lib().kf_gemm_dgrad_stacked_bf16(dy2.data_ptr(), *ptrs, out.data_ptr(), m, k, *rows, dy2.stride(0), pitch[0], k,
                                                sm_count(), _stream()), "kf_gemm_dgrad_stacked_bf16")
        return out
    return gemm(dy2, stack_rows(weights), a_kmajor=True, b_kmajor=False)


def swiglu_rows(x2: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor) -> torch.Tensor:
    """silu(x2 Wgᵀ) * (x2 Wuᵀ) without keeping the pre-activations."""
    m, k = x2.shape
    f = wg.shape[0]
    if m <= SKINNY_MAX_ROWS and f % 8 == 0 and k % 8 == 0:
        h = torch.empty((m, f), dtype=torch.bfloat16, device=x2.device)
        _check(lib().kf_gemm_skinny_swiglu_bf16(x2.data_ptr(), wg.data_ptr(), wu.data_ptr(), h.data_ptr(), m, f, k,
                                                x2.stride(0), wg.stride(0), wu.stride(0), f, 0, sm_count(), _stream()),
               "kf_gemm_skinny_swiglu_bf16")
        return h
    if gemm_swiglu_pair_supported(x2, wg, f) and wg.stride() == wu.stride():
        return gemm_swiglu_pair(x2, wg, wu, want_gu=False)[0]
    return swiglu_fwd(gemm_rows(x2, [wg, wu]))


def rope_tables_ok(cos: torch.Tensor, sin: torch.Tensor) -> bool:
    """The kernels with the rotation in their epilogue read fp32 tables 16 bytes at a time; tables that start elsewhere (slices
    of a packed buffer) are left to the separate rotary kernel, which reads single values."""
    return (cos.dtype == torch.float32 and sin.dtype == torch.float32 and cos.is_contiguous() and sin.is_contiguous()
            and (cos.data_ptr() | sin.data_ptr()) % 16 == 0)


def _gemm_rope(x2: torch.Tensor, weights, out: torch.Tensor, rope: tuple) -> torch.Tensor:
    cos, sin, seq_len, rope_cols, hd = rope
    m, k = x2.shape
    assert out.dtype == torch.bfloat16
    assert rope_tables_ok(cos, sin)
    assert cos.shape[-1] == hd // 2 and cos.numel() >= seq_len * (hd // 2) and m % seq_len == 0
    ptrs, rows, pitch = _weights3(weights)
    _check(lib().kf_gemm_rope_bf16(x2.data_ptr(), *ptrs, out.data_ptr(), m, *rows, k, x2.stride(0), pitch[0], out.stride(0),
                                   cos.data_ptr(), sin.data_ptr(), int(seq_len), int(rope_cols), int(hd), sm_count(), _stream()),
           "kf_gemm_rope_bf16")
    return out


def qkv_rope(x2: torch.Tensor, weights, cos, sin, s: int, hd: int) -> torch.Tensor:
    """Fused q | k | v projection (M, (H + 2 Hkv) hd) of M = B * s rows with q and k rotated by position ``row % s``."""
    wq, wk, wv = weights
    m = x2.shape[0]
    n = wq.shape[0] + wk.shape[0] + wv.shape[0]
    rope_cols = wq.shape[0] + wk.shape[0]
    if (m > SKINNY_MAX_ROWS and gemm_rope_supported(x2, wq, hd) and rope_tables_ok(cos, sin) and wk.shape[0] % hd == 0 and n % 256 == 0
            and wq.stride() == wk.stride() == wv.stride()
            and (rows_adjacent(weights) or (wq.shape[0] % 128 == 0 and wk.shape[0] % 128 == 0))):
        out = torch.empty((m, n), dtype=torch.bfloat16, device=x2.device)
        ws = [stack_rows(weights)] if rows_adjacent(weights) else weights
        return _gemm_rope(x2, ws, out, (cos, sin, s, rope_cols, hd))
    qkv = gemm_rows(x2, weights)
    qkv4 = qkv.view(m // s, s, n // hd, hd)
    rope(qkv4, cos, sin, rope_cols // hd, inverse=False, out=qkv4)
    return qkv


def block_decode(y: torch.Tensor, attn_ptrs, mlp_ptrs, cache_ptrs, table_ptrs, dims, scalars, foreign=None) -> None:
    """One new token per sequence through a block (``mlp_ptrs`` None: its attention half) as one native call.  ``y`` (B, 1, D)
    receives the output; k and v of the new position go into the cache.  The pointers and sizes are those of
    ``kf_block_decode_bf16``, handed over as two arrays (32 separate arguments cost ctypes more than the launches' set-up).

    Attention runs on the kernel split over the cache for head dim 128.  With head dim 64 it stays on what the op-by-op path
    uses: the 128-row tile kernel for one sequence, ``foreign(q)`` (rows of H hd) -> dense (B, H hd) between two native calls
    for more.  The reason is that a small model's logits stay bit for bit the same, not
    speed.  Measured (12 heads of 64, one query head per KV head, us, at 300 / 1000 / 2000 / 4000 positions): one sequence, split
    kernel 5.2 / 6.3 / 7.7 / 10.1, tile kernel 7.7 / 12.3 / 19.7 / 34.7, library 4.9 / 6.5 / 7.9 / 8.8; four sequences, split
    6.1 / 8.2 / 11.1 / 17.3, library 5.4 / 7.2 / 9.6 / 14.6; sixteen, split 9.7 / 18.9 / 31.2 / 54.8, library 9.2 / 16.9 / 25.6 /
    40.4."""
    b, d, h, hkv, hd, f = dims[:6]
    tile = hd == 64 and b == 1
    qc = h * hd
    # one buffer for all intermediates: n (D) | q (H hd) | hidden (F) | h1 (D) | attention (H hd) | rstd, lse
    scratch = torch.empty(b * (2 * d + 2 * qc + f) + 2 * b + 2 * h, dtype=torch.bfloat16, device=y.device)
    base = scratch.data_ptr()
    att = base + 2 * b * (2 * d + qc + f)
    rstd = att + 2 * b * qc
    yp = y.data_ptr()
    h1 = base + 2 * b * (d + qc + f) if mlp_ptrs else yp
    ints = array("q", (*attn_ptrs, *(mlp_ptrs or (0, 0, 0, 0)), *cache_ptrs, base, rstd, h1, yp, *table_ptrs, *dims, sm_count(),
                       7, int(tile), att, rstd + 4 * b))
    reals = array("d", scalars)
    fn, ip, rp = lib().kf_block_decode_bf16, ints.buffer_info()[0], reals.buffer_info()[0]
    norms = 0 if b <= lib().kf_skinny_norm_rows() else 1   # norm kernels per half of the block
    if hd == 64 and b > 1:
        ints[27] = 1
        _check(fn(ip, rp, _stream()), "kf_block_decode_bf16", 1 + norms)
        out = foreign(scratch[b * d : b * (d + qc)].view(b, qc))
        ints[27], ints[29] = 4, out.data_ptr()
        _check(fn(ip, rp, _stream()), "kf_block_decode_bf16", 3 + norms if mlp_ptrs else 1)
        return
    _check(fn(ip, rp, _stream()), "kf_block_decode_bf16", 5 + 2 * norms if mlp_ptrs else 3 + norms)


_steps = None   # the module once it is loaded, False when there is none for this Python and PyTorch


def _load_steps():
    """The CPython module of ``csrc/steps.cpp``, told the classes it looks for and the native entry.  False when there is none for this
    Python and PyTorch (its name holds both): the rules in Python (``fused_infer._plan``) then serve every call, with the same kernels."""
    global _steps
    if not STEPS_PATH.exists():
        get_logger(__name__).warning("%s is missing: generation steps are checked in Python (run `python -m kempnerforge_b200.ops.build`)",
                                     STEPS_PATH)
        _steps = False
        return _steps
    from kempnerforge_b200.models.attention import Attention, KVCache
    from kempnerforge_b200.models.mlp import SwiGLUMLP
    from kempnerforge_b200.models.norm import RMSNorm

    spec = importlib.util.spec_from_file_location("kf_steps", STEPS_PATH)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    mod.configure(Attention, SwiGLUMLP, RMSNorm, KVCache, torch.nn.Parameter,
                  ctypes.cast(lib().kf_blocks_decode_bf16, c_void_p).value, SKINNY_MAX_ROWS, lib().kf_skinny_norm_rows())
    _steps = mod
    return mod


def blocks_decode(blocks: list, caches: list, x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, foreign=None):
    """One new token per sequence through a row of plain blocks (attention on our kernels and a SwiGLU MLP) as one native call that
    checks them as well (``csrc/steps.cpp``): the last block's output (B, 1, D), or None when one of them is not plainly
    covered.  Without ``foreign`` the call stands for the blocks themselves, so hooks on them count; a block that calls it
    gives its ``foreign(q (B, H hd), H, hd, position)`` -> (B, H hd) for the attention of heads of 64 over several sequences."""
    steps = _load_steps() if _steps is None else _steps
    r = steps.decode(blocks, caches, x, cos, sin, foreign, _stream(), sm_count()) if steps else None
    if r is None:
        return None
    if type(r) is int:
        raise NativeKernelError(f"kf_blocks_decode_bf16 failed with code {r}")
    global LAUNCH_COUNT
    LAUNCH_COUNT += r[1]
    return r[0]


# --------------------------------------------------------------------------- norm / rope / swiglu / embedding
def rmsnorm_fwd(x: torch.Tensor, w: torch.Tensor, eps: float):
    rows, d = x.shape
    y = torch.empty_like(x)
    rstd = torch.empty(rows, dtype=torch.float32, device=x.device)
    _check(
        lib().kf_rmsnorm_fwd_bf16(x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr(), rows, d, eps, _stream()),
        "kf_rmsnorm_fwd_bf16",
    )
    return y, rstd


def rmsnorm_bwd(dy, x, w, rstd, residual_grad: torch.Tensor | None = None, out: torch.Tensor | None = None,
                dw_out: torch.Tensor | None = None):
    """Returns (dx, dw).  ``residual_grad`` is added to dx inside the kernel (it may be the same tensor as ``out``)."""
    rows, d = x.shape
    nb = lib().kf_rmsnorm_bwd_blocks(rows)
    partial = torch.empty(nb * d, dtype=torch.float32, device=x.device)
    dx = out if out is not None else torch.empty_like(x)
    dw = dw_out if dw_out is not None else torch.empty(d, dtype=torch.bfloat16, device=x.device)
    _check(
        lib().kf_rmsnorm_bwd_bf16(
            dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr(), dx.data_ptr(), partial.data_ptr(),
            dw.data_ptr(), None, rows, d, residual_grad.data_ptr() if residual_grad is not None else None, _stream(),
        ),
        "kf_rmsnorm_bwd_bf16",
    )
    return dx, dw


def cache_rows(kv: torch.Tensor, k: torch.Tensor, v: torch.Tensor, s: int) -> None:
    """k[:, :s], v[:, :s] = the halves of kv (B * s, 2 * Hkv * hd), rows at any pitch, for contiguous bf16 caches (B, max_len, Hkv, hd)."""
    b, width = k.shape[0], k.shape[2] * k.shape[3]
    assert kv.shape == (b * s, 2 * width) and kv.stride(1) == 1 and k.shape == v.shape and s <= k.shape[1]
    assert kv.dtype == k.dtype == v.dtype == torch.bfloat16 and k.is_contiguous() and v.is_contiguous() and kv.device == k.device == v.device
    _check(lib().kf_cache_rows_bf16(kv.data_ptr(), kv.stride(0), k.data_ptr(), v.data_ptr(), b, s, width, k.stride(0), _stream()),
           "kf_cache_rows_bf16")


def rope(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, n_rot: int, inverse: bool, out=None):
    b, s, h, hd = x.shape
    y = torch.empty_like(x) if out is None else out
    assert cos.dtype == torch.float32 and cos.shape[0] >= s and cos.shape[1] == hd // 2
    cos, sin = cos.contiguous(), sin.contiguous()   # the kernel steps from row to row by the width
    _check(
        lib().kf_rope_bf16(x.data_ptr(), y.data_ptr(), cos.data_ptr(), sin.data_ptr(), b * s, s, h, n_rot, hd, int(inverse), _stream()),
        "kf_rope_bf16",
    )
    return y


def swiglu_fwd(gu: torch.Tensor) -> torch.Tensor:
    h = gu.shape[-1] // 2
    rows = gu.numel() // (2 * h)
    out = torch.empty((*gu.shape[:-1], h), dtype=gu.dtype, device=gu.device)
    _check(lib().kf_swiglu_fwd_bf16(gu.data_ptr(), out.data_ptr(), rows, h, _stream()), "kf_swiglu_fwd_bf16")
    return out


def swiglu_bwd(dh: torch.Tensor, gu: torch.Tensor, out=None) -> torch.Tensor:
    h = gu.shape[-1] // 2
    rows = gu.numel() // (2 * h)
    dgu = torch.empty_like(gu) if out is None else out
    _check(lib().kf_swiglu_bwd_bf16(dh.data_ptr(), gu.data_ptr(), dgu.data_ptr(), rows, h, _stream()), "kf_swiglu_bwd_bf16")
    return dgu


def embedding_fwd(ids: torch.Tensor, table: torch.Tensor) -> torch.Tensor:
    ids = ids.contiguous()
    if ids.dtype != torch.int64:
        ids = ids.long()
    v, d = table.shape
    out = torch.empty((*ids.shape, d), dtype=table.dtype, device=table.device)
    _check(lib().kf_embedding_fwd_bf16(ids.data_ptr(), table.data_ptr(), out.data_ptr(), ids.numel(), d, v, _stream()), "kf_embedding_fwd_bf16")
    return out


def embedding_bwd(dy: torch.Tensor, ids: torch.Tensor, dtable: torch.Tensor, accumulate: bool) -> None:
    ids = ids.contiguous()
    if ids.dtype != torch.int64:
        ids = ids.long()
    v, d = dtable.shape
    if not accumulate:
        dtable.zero_()
    _check(lib().kf_embedding_bwd_bf16(ids.data_ptr(), dy.data_ptr(), dtable.data_ptr(), ids.numel(), d, v, _stream()), "kf_embedding_bwd_bf16")


# --------------------------------------------------------------------------- cross entropy
# Row statistics in the epilogue of the logits pay where its exponentials hide behind the products (K) and where a second read of the rows
# comes from HBM rather than from the 126 MB of L2 (bytes of logits).  Product and cross entropy, us, without / with: 2047 x 128 256 from
# 4096 1613 / 1548, 1024 x 128 256 from 2048 490 / 454, 4096 x 32 000 from 2048 455 / 440 and from 1024 288 / 281, 4096 x 50 304 from 1024
# 449 / 430; the whole loss over 1698 rows from 768 341 / 344, over 249 rows of 128 256 from 4096 949 / 952.
LOGITS_MIN_K = 1024
LOGITS_MIN_BYTES = 128 << 20


def gemm_logits(h: torch.Tensor, weight: torch.Tensor):
    """(:func:`gemm` of K-major operands, for every tile of its columns and row the largest value and the sum of exponentials relative to
    it as (tiles, rows, 2) fp32, or None where another kernel makes the product)."""
    (m, k), n = h.shape, weight.shape[0]
    width = 0
    if GEMM_MODE == 0 and k >= LOGITS_MIN_K and 2 * m * n >= LOGITS_MIN_BYTES and not _few_rows(m, n) and k % 8 == 0 and h.stride(0) % 8 == 0 and weight.stride(0) % 8 == 0:
        width = lib().kf_gemm_logits_width(m, n, k, sm_count())
    if width == 0 or h.data_ptr() % 16 or weight.data_ptr() % 16:
        return gemm(h, weight, a_kmajor=True, b_kmajor=True), None
    assert h.dtype == weight.dtype == torch.bfloat16 and weight.shape[1] == k and h.stride(1) == weight.stride(1) == 1
    assert h.device == weight.device
    out = torch.empty((m, n), dtype=torch.bfloat16, device=h.device)
    stats = torch.empty((-(-n // width), m, 2), dtype=torch.float32, device=h.device)
    _check(lib().kf_gemm_logits_bf16(h.data_ptr(), weight.data_ptr(), out.data_ptr(), stats.data_ptr(), m, n, k, h.stride(0), weight.stride(0), n,
                                     sm_count(), _stream()), "kf_gemm_logits_bf16")
    return out, stats


def ce_fwd_bwd(logits: torch.Tensor, labels: torch.Tensor, stats: torch.Tensor, inv_n: torch.Tensor, z_weight: float,
               tiles: torch.Tensor | None = None) -> None:
    """Overwrites ``logits`` (rows, V) with d loss / d logits and adds [sum nll, sum lse²] into ``stats``.  ``tiles``: what
    :func:`gemm_logits` returned with them."""
    rows, v = logits.shape
    assert logits.stride(1) == 1
    row_nll = torch.empty(rows, dtype=torch.float32, device=logits.device)
    row_lse2 = torch.empty(rows, dtype=torch.float32, device=logits.device)
    labels = labels.contiguous()
    if tiles is not None:
        row_lse = torch.empty(rows, dtype=torch.float32, device=logits.device)
        _check(lib().kf_ce_grad_bf16(logits.data_ptr(), tiles.data_ptr(), tiles.shape[0], labels.data_ptr(), row_lse.data_ptr(),
                                     row_nll.data_ptr(), row_lse2.data_ptr(), inv_n.data_ptr(), float(z_weight), rows, v, logits.stride(0),
                                     _stream()), "kf_ce_grad_bf16", 2)
    else:
        _check(
            lib().kf_ce_fwd_bwd_bf16(
                logits.data_ptr(), labels.data_ptr(), row_nll.data_ptr(), row_lse2.data_ptr(), inv_n.data_ptr(),
                float(z_weight), rows, v, logits.stride(0), _stream(),
            ),
            "kf_ce_fwd_bwd_bf16",
        )
    stats[0] += row_nll.sum()
    stats[1] += row_lse2.sum()


def scale_(x: torch.Tensor, factor: torch.Tensor) -> torch.Tensor:
    """x *= factor in place (contiguous bf16 x, one fp32 device scalar); costs nothing on the device when it is one."""
    assert x.is_contiguous() and x.dtype == torch.bfloat16 and factor.dtype == torch.float32 and factor.numel() == 1
    _check(lib().kf_scale_bf16(x.data_ptr(), x.numel(), factor.data_ptr(), _stream()), "kf_scale_bf16")
    return x


# --------------------------------------------------------------------------- optimizer
_DT = {torch.bfloat16: 0, torch.float32: 1}


# A kernel writes through an address, which what is kept by a tensor's version (fp8 copies of weights) does not see.  A flat buffer's version
# is moved; a parameter's own is not, because graphs that hold the parameter would be refused by it: it carries a count.
_wrote_buffer = torch.autograd.graph.increment_version


def _wrote_parameter(p: torch.Tensor) -> None:
    p._kf_writes = getattr(p, "_kf_writes", 0) + 1


def adamw_flat(p, g, m, v, n_decay: int, lr: float, beta1: float, beta2: float, eps: float, wd: float,
               step: int, grad_scale: torch.Tensor | None = None, skip: torch.Tensor | None = None) -> None:
    """One fused AdamW update over flat 1-D buffers; elements [0, n_decay) are weight-decayed."""
    n = p.numel()
    bc1 = 1.0 - beta1**step
    bc2_sqrt = math.sqrt(1.0 - beta2**step)
    _check(
        lib().kf_adamw_flat(
            p.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), n, n_decay, lr, beta1, beta2, eps, wd,
            bc1, bc2_sqrt, grad_scale.data_ptr() if grad_scale is not None else None,
            skip.data_ptr() if skip is not None else None, _DT[p.dtype], _DT[g.dtype], _DT[m.dtype], _stream(),
        ),
        "kf_adamw_flat",
    )
    _wrote_buffer(p)


def sumsq(x: torch.Tensor, out: torch.Tensor, accumulate: bool = False) -> torch.Tensor:
    """out[0] (+)= sum(x²) in fp32 with a fixed reduction order."""
    partial = torch.empty(1024, dtype=torch.float32, device=x.device)
    _check(lib().kf_sumsq(x.data_ptr(), x.numel(), _DT[x.dtype], partial.data_ptr(), out.data_ptr(), int(accumulate), _stream()), "kf_sumsq")
    return out


def gemm_swiglu(x2: torch.Tensor, w_gate_up: torch.Tensor, want_gu: bool = True):
    """(h, gu): h = silu(x Wgᵀ) * (x Wuᵀ) computed in the epilogue of one tcgen05 GEMM over the stacked weight
    ``w_gate_up`` = [Wg ; Wu] of shape (2F, K); ``gu`` (M, 2F) holds the pre-activations when ``want_gu``."""
    f = w_gate_up.shape[0] // 2
    return gemm_swiglu_pair(x2, w_gate_up[:f], w_gate_up[f:], want_gu)


def gemm_swiglu_pair(x2: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor, want_gu: bool = True):
    """:func:`gemm_swiglu` over a gate and an up weight (F, K) of one row pitch, read where they are."""
    m, k = x2.shape
    f = wg.shape[0]
    assert wg.shape == wu.shape and wg.stride() == wu.stride()
    h = torch.empty((m, f), dtype=torch.bfloat16, device=x2.device)
    gu = torch.empty((m, 2 * f), dtype=torch.bfloat16, device=x2.device) if want_gu else None
    _check(lib().kf_gemm_swiglu_bf16(x2.data_ptr(), wg.data_ptr(), wu.data_ptr(), h.data_ptr(),
                                     gu.data_ptr() if want_gu else None, m, f, k, x2.stride(0), wg.stride(0), f, 2 * f,
                                     sm_count(), _stream()),
           "kf_gemm_swiglu_bf16")
    return h, gu


def gemm_swiglu_bwd(dy2: torch.Tensor, w_down: torch.Tensor, gu: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    """d[gate | up] (M, 2F), written to ``out`` (default: over ``gu``): the input-gradient GEMM of the down projection (``dy2`` (M, K) times
    ``w_down`` (K, F) as stored) with the SwiGLU gradient in its epilogue; the gradient of the hidden activation is
    never written to memory."""
    m, k = dy2.shape
    f = w_down.shape[1]
    assert w_down.shape[0] == k and gu.shape == (m, 2 * f) and gu.is_contiguous() and w_down.stride(1) == 1
    out = gu if out is None else out
    assert out.shape == gu.shape and out.dtype == gu.dtype and out.is_contiguous()
    _check(lib().kf_gemm_swiglu_bwd_bf16(dy2.data_ptr(), w_down.data_ptr(), gu.data_ptr(), out.data_ptr(), m, f, k,
                                         dy2.stride(0), w_down.stride(0), 2 * f, sm_count(), _stream()),
           "kf_gemm_swiglu_bwd_bf16")
    return out


def gemm_symm(x: torch.Tensor, tall: bool = False, residual: torch.Tensor | None = None, alpha: float = 1.0,
              beta: float = 0.0, diag: float = 0.0) -> torch.Tensor:
    """bf16 (n, n) = alpha * x xᵀ + beta * residual + diag * I for x (n, K), or alpha * xᵀ x + ... for ``tall`` x (K, n).

    Only the tiles on and above the diagonal go through the tensor cores; the kernel stores each of them a second time
    transposed, so the result is exactly symmetric.  ``residual`` must be symmetric."""
    assert x.dtype == torch.bfloat16 and x.stride(1) == 1
    n, k = (x.shape[1], x.shape[0]) if tall else x.shape
    out = torch.empty((n, n), dtype=torch.bfloat16, device=x.device)
    if residual is not None:
        assert residual.shape == (n, n) and residual.dtype == torch.bfloat16 and residual.stride(1) == 1
    _check(lib().kf_gemm_symm_bf16(int(tall), x.data_ptr(), out.data_ptr(), residual.data_ptr() if residual is not None else None,
                                   n, k, x.stride(0), n, residual.stride(0) if residual is not None else 0, float(alpha),
                                   float(beta), float(diag), sm_count(), _stream()), "kf_gemm_symm_bf16")
    return out


def gemm_symm_supported(x: torch.Tensor, tall: bool = False) -> bool:
    n, k = (x.shape[1], x.shape[0]) if tall else x.shape
    return (getattr(lib(), "kf_gemm_symm_bf16", None) is not None and os.environ.get("KF_GEMM_SYMM", "1") == "1"
            and x.dtype == torch.bfloat16 and x.stride(1) == 1 and x.stride(0) % 8 == 0 and n % 8 == 0 and n >= 256
            and k % 64 == 0)


def gemm_swiglu_bwd_supported(dy2: torch.Tensor, w_down: torch.Tensor, gu: torch.Tensor | None) -> bool:
    return (gu is not None and getattr(lib(), "kf_gemm_swiglu_bwd_bf16", None) is not None
            and not os.environ.get("KF_DISABLE_SWIGLU_EPILOGUE") and os.environ.get("KF_SWIGLU_BWD_EPILOGUE", "1") == "1" and dy2.shape[0] >= 256 and dy2.shape[1] % 64 == 0
            and w_down.shape[1] % 256 == 0 and dy2.stride(0) % 8 == 0 and w_down.stride(0) % 8 == 0 and gu.is_contiguous()
            and dy2.dtype == torch.bfloat16)


def gemm_swiglu_supported(x2: torch.Tensor, w_gate_up: torch.Tensor) -> bool:
    return gemm_swiglu_pair_supported(x2, w_gate_up, w_gate_up.shape[0] // 2)


def gemm_swiglu_pair_supported(x2: torch.Tensor, w: torch.Tensor, f: int) -> bool:
    """``f`` hidden units; ``w``: the gate weight (the up weight has its strides) or both stacked."""
    return (getattr(lib(), "kf_gemm_swiglu_bf16", None) is not None and not os.environ.get("KF_DISABLE_SWIGLU_EPILOGUE")
            and f % 128 == 0 and x2.shape[0] >= 256 and x2.stride(1) == 1 and w.stride(1) == 1
            and x2.stride(0) % 8 == 0 and w.stride(0) % 8 == 0 and x2.dtype == torch.bfloat16)


# --------------------------------------------------------------------------- fp8
class PartialMax(NamedTuple):
    """Where |x| was taken the maximum of: a slot for the scale that :func:`fp8_cast` makes of it, then ``count`` partial maxima."""

    scratch: torch.Tensor
    count: int


def fp8_absmax(x2: torch.Tensor) -> PartialMax:
    """The maxima that :func:`fp8_scale` makes its scale of."""
    scratch = torch.empty(1 + 1024, dtype=torch.float32, device=x2.device)
    if not x2.is_contiguous():
        x2 = x2.contiguous()
    count = ctypes.c_int()
    _check(lib().kf_fp8_absmax_bf16(x2.data_ptr(), x2.numel(), scratch.data_ptr() + 4, ctypes.byref(count), _stream()), "kf_fp8_absmax_bf16")
    return PartialMax(scratch, count.value)


def fp8_scale(x2: torch.Tensor, e5m2: bool = False) -> torch.Tensor:
    """Device scalar fp8_max / absmax(x) (fp32, shape (1,)), for callers that want the scale itself; the fp8 layers leave it to
    :func:`fp8_cast`."""
    scratch = torch.empty(1 + 1024, dtype=torch.float32, device=x2.device)   # the scale, then partial maxima
    if not x2.is_contiguous():
        x2 = x2.contiguous()
    _check(lib().kf_fp8_scale_bf16(x2.data_ptr(), x2.numel(), int(e5m2), scratch[1:].data_ptr(), scratch.data_ptr(),
                                   _stream()), "kf_fp8_scale_bf16")
    return scratch[:1]


def fp8_cast(x2: torch.Tensor, scale: torch.Tensor | PartialMax, e5m2: bool, want_row: bool = True, want_t: bool = False):
    """fp8 bytes of x * scale: (rows, cols) and / or the transposed (cols, rows) copy, as uint8 tensors.  The rows of the transposed
    copy start on 128 bytes.  Of the maxima of x the kernel makes the scale itself and leaves it in ``scratch[:1]``."""
    partial, count = None, 0
    if isinstance(scale, PartialMax):
        partial, count, scale = scale.scratch.data_ptr() + 4, scale.count, scale.scratch
    rows, cols = x2.shape
    assert x2.stride(1) == 1
    row = torch.empty((rows, cols), dtype=torch.uint8, device=x2.device) if want_row else None
    # A product over the rows of x reads 128 bytes of every row of the copy at a time: at a pitch of 2000 each of those reads spans two
    # lines.  Weight gradients of a 7B feed-forward over 2000 tokens, us: gate | up 216 -> 151, down 107 -> 77
    pitch = -(-rows // 128) * 128
    t = torch.empty((cols, pitch), dtype=torch.uint8, device=x2.device)[:, :rows] if want_t else None
    _check(lib().kf_fp8_cast_bf16(x2.data_ptr(), rows, cols, x2.stride(0), partial, count, scale.data_ptr(), int(e5m2),
                                  row.data_ptr() if want_row else None, cols, t.data_ptr() if want_t else None, pitch,
                                  _stream()), "kf_fp8_cast_bf16")
    return row, t


def gemm_fp8(a8: torch.Tensor, b8: torch.Tensor, sa: torch.Tensor, sb: torch.Tensor, a_e5m2: bool = False,
             b_e5m2: bool = False, out: torch.Tensor | None = None, accumulate: bool = False) -> torch.Tensor:
    """bf16 (M, N) = a8 (M, K) @ b8 (N, K)ᵀ / (sa * sb) on the fp8 tensor cores."""
    m, k = a8.shape
    n = b8.shape[0]
    assert b8.shape[1] == k and a8.stride(1) == 1 and b8.stride(1) == 1
    if out is None:
        out = torch.empty((m, n), dtype=torch.bfloat16, device=a8.device)
        accumulate = False
    assert out.stride(1) == 1
    _check(lib().kf_gemm_fp8(a8.data_ptr(), b8.data_ptr(), out.data_ptr(), m, n, k, a8.stride(0), b8.stride(0),
                             out.stride(0), int(a_e5m2), int(b_e5m2), sa.data_ptr(), sb.data_ptr(), int(accumulate),
                             sm_count(), _stream()), "kf_gemm_fp8")
    return out


def gemm_fp8_swiglu(a8: torch.Tensor, b8: torch.Tensor, sa: torch.Tensor, sb: torch.Tensor, want_gu: bool = True):
    """(gu or None, h, maxima of h): :func:`gemm_fp8` of e4m3 operands, b8 = [gate ; up] (2F rows), :func:`swiglu_fwd` of it and
    :func:`fp8_absmax` of that, from one kernel."""
    m, k = a8.shape
    f = b8.shape[0] // 2
    assert b8.shape == (2 * f, k) and a8.stride(1) == 1 and b8.stride(1) == 1
    gu = torch.empty((m, 2 * f), dtype=torch.bfloat16, device=a8.device) if want_gu else None
    h = torch.empty((m, f), dtype=torch.bfloat16, device=a8.device)
    scratch = torch.empty(1 + 8 * sm_count(), dtype=torch.float32, device=a8.device)
    count = ctypes.c_int()
    _check(lib().kf_gemm_fp8_swiglu(a8.data_ptr(), b8.data_ptr(), h.data_ptr(), _ptr(gu), m, f, k, a8.stride(0), b8.stride(0), f, 2 * f,
                                    sa.data_ptr(), sb.data_ptr(), scratch.data_ptr() + 4, ctypes.byref(count), sm_count(), _stream()),
           "kf_gemm_fp8_swiglu")
    return gu, h, PartialMax(scratch, count.value)


def gemm_fp8_swiglu_bwd(a8: torch.Tensor, b8: torch.Tensor, sa: torch.Tensor, sb: torch.Tensor, gu: torch.Tensor):
    """(dgu, its maxima): :func:`swiglu_bwd` of :func:`gemm_fp8` of an e5m2 gradient and e4m3 weights (F rows) in a tensor of its own,
    and :func:`fp8_absmax` of it; the gradient of the hidden activation stays on the chip."""
    m, k = a8.shape
    f = b8.shape[0]
    assert b8.shape[1] == k and a8.stride(1) == 1 and b8.stride(1) == 1 and gu.shape == (m, 2 * f)
    if not gu.is_contiguous() or gu.data_ptr() % 32:
        gu = gu.clone(memory_format=torch.contiguous_format)
    dgu = torch.empty_like(gu)
    scratch = torch.empty(1 + 8 * sm_count(), dtype=torch.float32, device=a8.device)
    count = ctypes.c_int()
    _check(lib().kf_gemm_fp8_swiglu_bwd(a8.data_ptr(), b8.data_ptr(), gu.data_ptr(), dgu.data_ptr(), m, f, k, a8.stride(0), b8.stride(0), 2 * f,
                                        sa.data_ptr(), sb.data_ptr(), scratch.data_ptr() + 4, ctypes.byref(count), sm_count(), _stream()),
           "kf_gemm_fp8_swiglu_bwd")
    return dgu, PartialMax(scratch, count.value)


# --------------------------------------------------------------------------- attention
def attn_policy() -> str:
    """``KF_ATTN``: "native" (default) = the tcgen05 kernels wherever they apply (training blocks included; shapes
    they do not cover fall back to the library call); "library" = never."""
    v = os.environ.get("KF_ATTN", "native")
    return "native" if v == "auto" else v


def _attn_rows_ok(t: torch.Tensor) -> bool:
    """(B, S, heads, hd) whose (b, s) pairs form evenly pitched rows with the heads side by side."""
    b, s, _, hd = t.shape
    return (t.stride(-1) == 1 and t.stride(2) == hd and (b == 1 or t.stride(0) == s * t.stride(1))
            and t.stride(1) % 8 == 0 and t.data_ptr() % 16 == 0)


def attn_supported(q, k, v, causal: bool, needs_grad: bool = False, docs: bool = False) -> bool:
    """Shapes the tcgen05 attention kernels cover: bf16, head dim 64 or 128, grouped KV heads, causal or full,
    optional document ids; q / k / v may be strided views of one fused projection output."""
    L = lib()
    if getattr(L, "kf_attn_fwd_bf16", None) is None or attn_policy() == "library":
        return False
    if needs_grad and (getattr(L, "kf_attn_bwd_bf16", None) is None
                       or not attn_bwd_chosen(q.shape[-1], q.shape[0] * q.shape[2], q.shape[1], k.shape[1], causal, docs)):
        return False
    if q.dtype != torch.bfloat16 or q.shape[-1] not in (64, 128) or q.shape[2] % k.shape[2] != 0:
        return False
    if causal and q.shape[1] != k.shape[1]:
        return False
    return _attn_rows_ok(q) and _attn_rows_ok(k) and _attn_rows_ok(v)


HEAD64_MAX_SCORES = 1 << 25
HEAD64_MAX_PARTS = 9 << 22   # 151 MB of dQ parts: what HEAD64_MAX_SCORES causal scores need, with a margin for whole tiles


def attn_bwd_chosen(hd: int, heads: int, sq: int, sk: int, causal: bool, docs: bool) -> bool:
    """Whether a fused node runs attention with gradients (``heads`` = batch x query heads) on the native kernels.  Head dim 128:
    always.  64: not with document ids, whose scores and probabilities the reference formulas hold in fp32; else up to
    ``HEAD64_MAX_SCORES`` visible scores (many sequences shorter than a tile: ``HEAD64_MAX_PARTS`` of scratch), and a program that asked for deterministic algorithms keeps the library, which knows of
    that.  Measured, forward + backward, us, native / library (12 causal heads): 100 positions 20 / 21, 3 x 333 34 / 30, 2048 101 /
    66, 4 x 2048 259 / 151.  Around the library's kernels a block also makes three copies and a rotation of q | k | v gradients and
    issues a second autograd graph from the host (170 us), which decides up to about the limit."""
    if hd != 64:
        return hd == 128
    return (not docs and heads * sq * sk // (2 if causal else 1) <= HEAD64_MAX_SCORES
            and attn_bwd_dq_floats(1, sq, sk, heads, hd) <= HEAD64_MAX_PARTS and not torch.are_deterministic_algorithms_enabled())


def doc_blocks(doc_ids: torch.Tensor, like: torch.Tensor | None = None):
    """(int32 ids (B, S), int32 (B, ceil(S / 64), 2) smallest and largest id of every 64 positions): what the attention
    kernels read of a document mask.  Pass the pair in place of the ids to reuse it for the backward.  ``like`` (B, S, ..): the
    keys they belong to; ids of as many positions in another shape and one row for all sequences are taken, any others refused."""
    ids = doc_ids if doc_ids.dtype in (torch.int32, torch.int64) else doc_ids.to(torch.int32)
    if like is not None:
        assert ids.device == like.device, f"document ids on {ids.device}, keys on {like.device}"
        if ids.shape != like.shape[:2]:
            ids = ids.reshape(like.shape[:2]) if ids.numel() == like.shape[0] * like.shape[1] else ids.expand(like.shape[:2])
    ids = ids.contiguous()
    b, s = ids.shape
    out = torch.empty((b, s), dtype=torch.int32, device=ids.device)
    rng = torch.empty((b, (s + 63) // 64, 2), dtype=torch.int32, device=ids.device)
    _check(lib().kf_doc_blocks(ids.data_ptr(), int(ids.dtype == torch.int64), out.data_ptr(), rng.data_ptr(), b, s, _stream()),
           "kf_doc_blocks")
    return out, rng


def attn_fwd(q, k, v, causal: bool, doc_ids, scale: float):
    """q (B, Sq, H, hd), k / v (B, Sk, Hkv, hd) -> out (B, Sq, H, hd) bf16 and lse (B, H, Sq) fp32.  ``doc_ids``: (B, Sk)
    ids, or what :func:`doc_blocks` made of them."""
    b, sq, h, hd = q.shape
    sk, hkv = k.shape[1], k.shape[2]
    out = torch.empty((b, sq, h, hd), dtype=q.dtype, device=q.device)
    lse = torch.empty((b, h, sq), dtype=torch.float32, device=q.device)
    doc = rng = None
    if doc_ids is not None:
        doc, rng = doc_ids if isinstance(doc_ids, tuple) else doc_blocks(doc_ids, k)
    # two query tiles per CTA (interleaved softmax) once there are at least two tiles; KF_ATTN_FWD=1 forces the
    # single-tile kernel
    L = lib()
    two = sq > 128 and getattr(L, "kf_attn_fwd2_bf16", None) is not None and os.environ.get("KF_ATTN_FWD", "2") != "1"
    fn = L.kf_attn_fwd2_bf16 if two else L.kf_attn_fwd_bf16
    mask = (_ptr(doc), _ptr(rng)) if two else (_ptr(doc),)
    _check(
        fn(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), *mask, b, sq, sk, h, hkv, hd, q.stride(1),
           k.stride(1), v.stride(1), h * hd, float(scale), int(causal), _stream()),
        "kf_attn_fwd2_bf16" if two else "kf_attn_fwd_bf16",
    )
    return out, lse


# --------------------------------------------------------------------------- Lion / schedule-free AdamW
def _same_flat(*ts: torch.Tensor) -> bool:
    d = ts[0].dtype
    return d in _DT and all(t.is_cuda and t.dtype == d and t.is_contiguous() and t.numel() == ts[0].numel() for t in ts)


def lion_step(p, g, m, lr: float, b1: float, b2: float, wd: float) -> bool:
    """In-place Lion update of one tensor; False when the tensors do not qualify (mixed dtypes, strided)."""
    if getattr(lib(), "kf_lion", None) is None or not _same_flat(p, g, m):
        return False
    _check(lib().kf_lion(p.data_ptr(), g.data_ptr(), m.data_ptr(), p.numel(), _DT[p.dtype], lr, b1, b2, wd, _stream()), "kf_lion")
    _wrote_parameter(p)
    return True


def sf_adamw_step(y, g, z, v, x, lr, b1, b2, eps, wd, bc2, ck, first: bool) -> bool:
    """In-place schedule-free AdamW update: y is the tensor the model reads, z / x the base and averaged iterates."""
    if getattr(lib(), "kf_sf_adamw", None) is None or not _same_flat(y, g, z, v, x):
        return False
    _check(lib().kf_sf_adamw(y.data_ptr(), g.data_ptr(), z.data_ptr(), v.data_ptr(), x.data_ptr(), y.numel(), _DT[y.dtype],
                             lr, b1, b2, eps, wd, bc2, ck, int(first), _stream()), "kf_sf_adamw")
    _wrote_parameter(y)
    return True


# --------------------------------------------------------------------------- mixture of experts
def router_topk(logits: torch.Tensor, bias: torch.Tensor | None, sigmoid: bool, k: int, half: bool = False):
    """(weights fp32 (T, k), the same in bf16 or None, indices int64 (T, k), what :func:`router_bwd` needs of the bias or the
    counts, token counts fp32 (E), mean scores fp32 (E), mean logsumexp² fp32 (), balance fp32 ()): ``balance`` = E sum(counts /
    (T k) * mean) of softmax scores, 0 of sigmoid ones.  ``half``: also the bf16 weights.  ``bias``: fp32 or bf16 (E)."""
    t, e = logits.shape
    assert logits.is_contiguous() and logits.dtype in (torch.bfloat16, torch.float32)
    dev = logits.device
    idx = torch.empty((t, k), dtype=torch.int64, device=dev)
    w = torch.empty((t, k), dtype=torch.float32, device=dev)
    w16 = torch.empty((t, k), dtype=torch.bfloat16, device=dev) if half else None
    # tensors of their own: a program may change any of them in place
    counts, mean, keep = (torch.empty(e, dtype=torch.float32, device=dev) for _ in range(3))
    z, balance = (torch.empty((), dtype=torch.float32, device=dev) for _ in range(2))
    acc = torch.empty(2 * e + 2, dtype=torch.float32, device=dev)
    assert bias is None or (bias.shape == (e,) and bias.is_contiguous() and bias.dtype in (torch.bfloat16, torch.float32))
    _check(lib().kf_router_topk(logits.data_ptr(), 0 if logits.dtype == torch.bfloat16 else 1, _ptr(bias),
                                int(bias is not None and bias.dtype == torch.bfloat16), int(sigmoid), t, e, k,
                                idx.data_ptr(), w.data_ptr(), _ptr(w16), keep.data_ptr(), counts.data_ptr(), mean.data_ptr(), z.data_ptr(),
                                balance.data_ptr(), acc.data_ptr(), _stream()), "kf_router_topk")
    if t == 0:   # no token, no launch: means over nothing
        counts.zero_(), keep.zero_(), mean.fill_(float("nan")), z.fill_(float("nan")), balance.fill_(0.0 if sigmoid else float("nan"))
    return w, w16, idx, keep, counts, mean, z, balance


def router_bwd(logits, keep, sigmoid: bool, idx, w, dw, dmean, dz, dbalance, dbias_dtype: torch.dtype | None):
    """(dlogits, dbias or None) of :func:`router_topk`: ``dw`` (T, k) fp32 or bf16, ``dmean`` (E) of the mean scores, ``dz`` of the
    mean squared logsumexp and ``dbalance`` of the balancing loss, all fp32 (each may be None).  ``dbias_dtype``: fp32 or bf16,
    None for no gradient of the bias."""
    t, e = logits.shape
    k = idx.shape[1]
    dlogits = torch.empty_like(logits)
    dbias = partial = None
    if dbias_dtype is not None:
        dbias = torch.empty(e, dtype=dbias_dtype, device=logits.device)
        partial = torch.empty(592 * e, dtype=torch.float32, device=logits.device)
    _check(lib().kf_router_bwd(logits.data_ptr(), 0 if logits.dtype == torch.bfloat16 else 1, keep.data_ptr(), int(sigmoid),
                               idx.data_ptr(), w.data_ptr(), _ptr(dw), int(dw is not None and dw.dtype == torch.bfloat16),
                               _ptr(dmean), _ptr(dz), _ptr(dbalance), keep.data_ptr(), t, e, k, dlogits.data_ptr(), _ptr(dbias),
                               int(dbias_dtype == torch.bfloat16), _ptr(partial), _stream()), "kf_router_bwd",
           2 if dbias is not None else 1)
    return dlogits, dbias


def moe_capacity_mask(indices: torch.Tensor, num_experts: int, cap: int) -> torch.Tensor:
    """fp32 (T, k) mask: 1 for the first ``cap`` tokens (sequence order) of every (slot, expert) pair, else 0."""
    t, k = indices.shape
    assert indices.dtype == torch.int64 and indices.is_contiguous()
    keep = torch.empty((t, k), dtype=torch.float32, device=indices.device)
    _check(lib().kf_moe_capacity_mask(indices.data_ptr(), t, k, num_experts, int(cap), keep.data_ptr(), _stream()),
           "kf_moe_capacity_mask")
    return keep


def moe_sort(indices: torch.Tensor, num_experts: int):
    """Stable sort of the (token, k) assignments by expert: (offsets int32 (E + 1), row_of_slot int32, slot_of_row int32)."""
    flat = indices.reshape(-1)
    assert flat.dtype == torch.int64 and flat.is_contiguous()
    slots = flat.numel()
    nb = (slots + 1023) // 1024
    scratch = torch.empty(max(nb, 1) * num_experts, dtype=torch.int32, device=flat.device)
    offsets = torch.empty(num_experts + 1, dtype=torch.int32, device=flat.device)
    row_of_slot = torch.empty(slots, dtype=torch.int32, device=flat.device)
    slot_of_row = torch.empty(slots, dtype=torch.int32, device=flat.device)
    _check(lib().kf_moe_sort(flat.data_ptr(), slots, num_experts, scratch.data_ptr(), offsets.data_ptr(),
                             row_of_slot.data_ptr(), slot_of_row.data_ptr(), _stream()), "kf_moe_sort")
    return offsets, row_of_slot, slot_of_row


def moe_gather(x: torch.Tensor, slot_of_row: torch.Tensor, k: int) -> torch.Tensor:
    rows, cols = slot_of_row.numel(), x.shape[1]
    out = torch.empty((rows, cols), dtype=x.dtype, device=x.device)
    _check(lib().kf_moe_gather_bf16(x.data_ptr(), slot_of_row.data_ptr(), rows, k, cols, out.data_ptr(), _stream()),
           "kf_moe_gather_bf16")
    return out


def moe_combine(y: torch.Tensor, row_of_slot: torch.Tensor, w: torch.Tensor | None, tokens: int, k: int,
                plus: torch.Tensor | None = None) -> torch.Tensor:
    """(T, D) sum over the k rows of every token, weighted by ``w`` (T, k) fp32 or bf16, and ``plus`` (T, D) added to it."""
    cols = y.shape[1]
    out = torch.empty((tokens, cols), dtype=y.dtype, device=y.device)
    assert w is None or w.dtype in (torch.float32, torch.bfloat16)
    _check(lib().kf_moe_combine_bf16(y.data_ptr(), row_of_slot.data_ptr(), _ptr(w), int(w is not None and w.dtype == torch.bfloat16),
                                     _ptr(plus), tokens, k, cols, out.data_ptr(), _stream()), "kf_moe_combine_bf16")
    return out


def moe_combine_bwd(dout: torch.Tensor, y: torch.Tensor, slot_of_row: torch.Tensor, w: torch.Tensor, k: int):
    """(dy, dw) of the weighted :func:`moe_combine`; ``dw`` in the type of ``w`` (fp32 or bf16), in slot order."""
    rows, cols = y.shape
    assert w.dtype in (torch.float32, torch.bfloat16)
    dy = torch.empty_like(y)
    dw = torch.empty(rows, dtype=w.dtype, device=y.device)
    _check(lib().kf_moe_combine_bwd_bf16(dout.data_ptr(), y.data_ptr(), slot_of_row.data_ptr(), w.data_ptr(),
                                         int(w.dtype == torch.bfloat16), rows, k, cols, dy.data_ptr(), dw.data_ptr(), _stream()),
           "kf_moe_combine_bwd_bf16")
    return dy, dw


def grouped_swiglu(a: torch.Tensor, wg: torch.Tensor, wu: torch.Tensor, offsets: torch.Tensor, b_mn: bool,
                   want_gu: bool = True):
    """(h, gu): h = silu(a @ Wg_e) * (a @ Wu_e) over the ragged expert row ranges in ONE grouped GEMM (activation in
    its epilogue); ``gu`` (rows, 2F) keeps the bf16 pre-activations (gate | up) when ``want_gu``.  Weights (E, F, K)
    or, with ``b_mn``, (E, K, F).  Rows past ``offsets[E]`` are left untouched."""
    rows, k = a.shape
    e = wg.shape[0]
    f = wg.shape[2] if b_mn else wg.shape[1]
    assert wg.shape == wu.shape and wg.is_contiguous() and wu.is_contiguous() and a.stride(1) == 1
    h = torch.empty((rows, f), dtype=torch.bfloat16, device=a.device)
    gu = torch.empty((rows, 2 * f), dtype=torch.bfloat16, device=a.device) if want_gu else None
    _check(lib().kf_grouped_swiglu_bf16(a.data_ptr(), wg.data_ptr(), wu.data_ptr(), h.data_ptr(),
                                        gu.data_ptr() if gu is not None else None, offsets.data_ptr(), rows, e, f, k,
                                        a.stride(0), f, 2 * f, int(b_mn), sm_count(), _stream()), "kf_grouped_swiglu_bf16")
    return h, gu


def grouped_swiglu_supported(a: torch.Tensor, wg: torch.Tensor, b_mn: bool) -> bool:
    return getattr(lib(), "kf_grouped_swiglu_bf16", None) is not None and grouped_gemm_supported(a, wg, b_mn) \
        and not os.environ.get("KF_DISABLE_GROUPED_SWIGLU")


def grouped_swiglu_bwd(dy: torch.Tensor, w_down: torch.Tensor, gu: torch.Tensor, offsets: torch.Tensor, b_mn: bool,
                       out: torch.Tensor | None = None) -> torch.Tensor:
    """d[gate | up] (rows, 2F), written to ``out`` (default: over ``gu``): the input-gradient product of the experts' down projection
    (``dy`` (rows, K) times ``w_down``: (E, F, K), or (E, K, F) with ``b_mn``) with the SwiGLU gradient in its epilogue;
    the gradient of the hidden activation is never written to memory.  Rows past ``offsets[E]`` stay untouched."""
    rows, k = dy.shape
    e = w_down.shape[0]
    f = w_down.shape[2] if b_mn else w_down.shape[1]
    out = gu if out is None else out
    assert gu.shape == (rows, 2 * f) and gu.is_contiguous() and w_down.is_contiguous() and dy.stride(1) == 1
    assert out.shape == gu.shape and out.dtype == gu.dtype and out.is_contiguous()
    _check(lib().kf_grouped_swiglu_bwd_bf16(dy.data_ptr(), w_down.data_ptr(), gu.data_ptr(), out.data_ptr(), offsets.data_ptr(),
                                            rows, e, f, k, dy.stride(0), 2 * f, int(b_mn), sm_count(), _stream()),
           "kf_grouped_swiglu_bwd_bf16")
    return out


def grouped_swiglu_bwd_supported(dy: torch.Tensor, w_down: torch.Tensor, b_mn: bool) -> bool:
    return (getattr(lib(), "kf_grouped_swiglu_bwd_bf16", None) is not None and grouped_gemm_supported(dy, w_down, b_mn)
            and os.environ.get("KF_SWIGLU_BWD_EPILOGUE", "1") == "1" and not os.environ.get("KF_DISABLE_GROUPED_SWIGLU")
            and dy.shape[0] >= 256 and sm_count() >= 2)


def swiglu_bwd_ragged(dh: torch.Tensor, gu: torch.Tensor, offsets: torch.Tensor) -> torch.Tensor:
    """dgu (rows, 2F) of h = silu(gate) * up for the rows below ``offsets[-1]`` (a device int; later rows untouched)."""
    rows, f = dh.shape
    assert gu.shape == (rows, 2 * f) and dh.is_contiguous() and gu.is_contiguous()
    dgu = torch.empty_like(gu)
    _check(lib().kf_swiglu_bwd_ragged_bf16(dh.data_ptr(), gu.data_ptr(), dgu.data_ptr(), rows, offsets[-1:].data_ptr(), f,
                                           _stream()), "kf_swiglu_bwd_ragged_bf16")
    return dgu


def grouped_gemm(a: torch.Tensor, b: torch.Tensor, offsets: torch.Tensor, b_mn: bool, out: torch.Tensor | None = None,
                 accumulate: bool = False):
    """Ragged grouped GEMM: rows ``offsets[e]:offsets[e+1]`` of ``a`` (rows, K) are multiplied by expert e's matrix.
    ``b`` is (E, N, K) when ``b_mn`` is False and (E, K, N) when True; ``offsets`` is int32 (E + 1) on the device.
    ``accumulate``: add to ``out``."""
    rows, k = a.shape
    e = b.shape[0]
    n = b.shape[2] if b_mn else b.shape[1]
    assert (b.shape[1] if b_mn else b.shape[2]) == k and b.is_contiguous() and a.stride(1) == 1
    assert offsets.dtype == torch.int32 and offsets.numel() == e + 1
    if out is None:
        out = torch.empty((rows, n), dtype=torch.bfloat16, device=a.device)
    _check(lib().kf_grouped_gemm_acc_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), offsets.data_ptr(), rows, e, n, k,
                                          a.stride(0), out.stride(0), int(b_mn), int(accumulate), sm_count(), _stream()),
           "kf_grouped_gemm_acc_bf16")
    return out


def grouped_gemm_supported(a: torch.Tensor, b: torch.Tensor, b_mn: bool) -> bool:
    if getattr(lib(), "kf_grouped_gemm_bf16", None) is None or a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16:
        return False
    k = a.shape[1]
    n = b.shape[2] if b_mn else b.shape[1]
    return (b.shape[0] <= 256 and k % 8 == 0 and n % 8 == 0 and (not b_mn or k % 64 == 0) and a.stride(1) == 1
            and a.stride(0) % 8 == 0 and b.is_contiguous())


MAX_SEPARATE_EXPERTS = 32   # experts whose weights the grouped kernels read through a tensor map each
_GROUPED_PAIR = os.environ.get("KF_GROUPED_PAIR", "1") != "0"


def grouped_pair_tiles() -> bool:
    return _GROUPED_PAIR and sm_count() >= 2


def grouped_experts(kind: int, a: torch.Tensor, w, w2, offsets: torch.Tensor, n: int, b_mn: bool, out: torch.Tensor,
                    gu: torch.Tensor | None = None) -> torch.Tensor:
    """Grouped products over expert rows on CTA-pair tiles: 0 ``a @ W_e``; 1 ``silu(a @ W_e) * (a @ W2_e)`` (``gu``: receives
    the pre-activations); 2 the SwiGLU gradient of ``a @ W_e`` given ``gu``; 3 ``a[:, :K/2] @ W_e + a[:, K/2:] @ W2_e``.
    ``w`` / ``w2``: one packed (E, .., ..) tensor or a list with one matrix per expert, (N, K) or, ``b_mn``, (K, N)."""
    rows, k = a.shape
    separate = isinstance(w, (list, tuple))
    e = offsets.numel() - 1
    arr = (c_void_p * e) if separate else (c_void_p * 1)
    wp = arr(*[t.data_ptr() for t in w]) if separate else arr(w.data_ptr())
    w2p = None if w2 is None else arr(*[t.data_ptr() for t in w2]) if separate else arr(w2.data_ptr())
    _check(lib().kf_grouped_experts_bf16(kind, a.data_ptr(), wp, w2p, int(separate), out.data_ptr(), _ptr(gu), offsets.data_ptr(),
                                         rows, e, n, k, a.stride(0), out.stride(0), gu.stride(0) if gu is not None else 0,
                                         int(b_mn), sm_count(), _stream()), "kf_grouped_experts_bf16")
    return out


def grouped_wgrad(a: torch.Tensor, b: torch.Tensor, offsets: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    """Per-expert ``a_e^T @ b_e`` over the ragged row ranges ``offsets[e]:offsets[e+1]``: (E, a.shape[1], b.shape[1])
    in bf16.  The weight gradient of :func:`grouped_gemm`; experts without rows get zeros."""
    rows, m = a.shape
    n = b.shape[1]
    e = offsets.numel() - 1
    assert b.shape[0] == rows and a.stride(1) == 1 and b.stride(1) == 1 and offsets.dtype == torch.int32
    if out is None:
        out = torch.empty((e, m, n), dtype=torch.bfloat16, device=a.device)
    assert out.shape == (e, m, n) and out.is_contiguous() and out.dtype == torch.bfloat16
    _check(lib().kf_grouped_wgrad_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), offsets.data_ptr(), rows, e, m, n,
                                       a.stride(0), b.stride(0), sm_count(), _stream()), "kf_grouped_wgrad_bf16")
    return out


def grouped_wgrad_supported(a: torch.Tensor, b: torch.Tensor) -> bool:
    if os.environ.get("KF_GROUPED_WGRAD", "1") == "0":  # escape hatch: weight gradients through torch._grouped_mm
        return False
    if getattr(lib(), "kf_grouped_wgrad_bf16", None) is None or a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16:
        return False
    return (a.shape[0] > 0 and a.shape[1] % 8 == 0 and b.shape[1] % 8 == 0 and a.stride(1) == 1 and b.stride(1) == 1
            and a.stride(0) % 8 == 0 and b.stride(0) % 8 == 0)


def all_gather_gemm(x_shard: torch.Tensor, w: torch.Tensor, ctx, seq_len: int, out: torch.Tensor | None = None,
                    w_kn: bool = False) -> torch.Tensor:
    """out[T, N] = gather over the ranks of ``ctx`` (along the sequence) of x_shard[T/tp, K], times the weight: w is
    (N, K) or, with ``w_kn``, (K, N) (the layout the input-gradient GEMM of a row-parallel Linear needs).  The shard is
    pushed to the peers by copy warps of the GEMM kernel itself.  ``ctx`` is a ``comm.fused_tp.AgGemmContext``."""
    tl, k = x_shard.shape
    t = tl * ctx.world
    n = w.shape[1] if w_kn else w.shape[0]
    assert x_shard.stride(1) == 1 and w.stride(1) == 1 and (w.shape[0] if w_kn else w.shape[1]) == k
    if out is None:
        out = torch.empty((t, n), dtype=torch.bfloat16, device=x_shard.device)
    ctx.reserve(t, k)
    _check(
        lib().kf_ag_gemm_bf16(x_shard.data_ptr(), w.data_ptr(), ctx.stage_ptrs, ctx.flag_ptrs, out.data_ptr(), t, n, k,
                              seq_len, x_shard.stride(0), w.stride(0), out.stride(0), ctx.world, ctx.rank, ctx.next_call(),
                              int(w_kn), sm_count(), _stream()),
        "kf_ag_gemm_bf16",
    )
    return out


def gemm_reduce_scatter(x2: torch.Tensor, w: torch.Tensor, ctx, seq_len: int, out: torch.Tensor | None = None,
                        residual: torch.Tensor | None = None, w_kn: bool = False) -> torch.Tensor:
    """out[T/tp, D] = reduce-scatter over the ranks of ``ctx`` of x2[T, K_local] times the weight (+ residual): w is
    (D, K_local) or, with ``w_kn``, (K_local, D) (the input-gradient GEMM of a column-parallel Linear).  Tiles are pushed
    to their owners from the GEMM epilogue.  ``ctx`` is a ``comm.fused_tp.GemmRSContext``."""
    t, k = x2.shape
    d = w.shape[1] if w_kn else w.shape[0]
    assert x2.stride(1) == 1 and w.stride(1) == 1 and (w.shape[0] if w_kn else w.shape[1]) == k
    tl = t // ctx.world
    if out is None:
        out = torch.empty((tl, d), dtype=torch.bfloat16, device=x2.device)
    ctx.reserve(t, d)
    _check(
        lib().kf_gemm_rs_bf16(x2.data_ptr(), w.data_ptr(), ctx.stage_ptrs, ctx.flag_ptrs, out.data_ptr(),
                              residual.data_ptr() if residual is not None else None, t, d, k, seq_len, x2.stride(0),
                              w.stride(0), ctx.world, ctx.rank, ctx.next_call(), int(w_kn), sm_count(), _stream()),
        "kf_gemm_rs_bf16",
    )
    return out


def grouped_pair_mode(mode: int) -> None:
    """1: the ragged grouped GEMMs run on CTA-pair tiles (default); 0: single-CTA 128 x 256 tiles."""
    global _GROUPED_PAIR
    _GROUPED_PAIR = bool(mode)
    lib().kf_grouped_pair_mode(int(mode))


def attn_bwd_dq_mode(mode: int) -> int:
    """How the attention backward adds its dQ tiles to the fp32 accumulator: 0 = one ``red.global`` per element,
    1 = one bulk tensor reduction (TMA) per tile staged in shared memory (default, 1.75x faster on the 8B shape).
    Returns the previous mode.  ``KF_ATTN_BWD_DQ=red`` selects 0 at load time."""
    return int(lib().kf_attn_bwd_dq_mode(int(mode)))


def gemm_rope_supported(x2: torch.Tensor, w: torch.Tensor, hd: int) -> bool:
    """The rotary epilogue lives in the CTA-pair kernel: bf16, head dim 64 / 128 / 256, whole heads per weight."""
    return (getattr(lib(), "kf_gemm_rope_bf16", None) is not None and hd in (64, 128, 256) and w.shape[0] % hd == 0
            and x2.dtype == torch.bfloat16 and x2.stride(0) % 8 == 0 and w.stride(0) % 8 == 0)


def attn_bwd_dq_floats(b: int, sq: int, sk: int, h: int, hd: int) -> int:
    """fp32 values of dQ scratch: one accumulator, or for head dim 64 a part per tile of 128 keys."""
    return b * sq * h * hd if hd != 64 else -(-sk // 128) * b * h * (-(-sq // 64) * 64) * 64


def attn_bwd(dout, q, k, v, out, lse, causal: bool, doc_ids, scale: float, dq=None, dk=None, dv=None, rope=None):
    """Gradients of ``attn_fwd``.  ``dq`` / ``dk`` / ``dv`` may be preallocated (strided) destinations, e.g. the
    three head ranges of one fused projection gradient; otherwise contiguous tensors are returned.
    ``rope = (cos, sin)`` (fp32 (S, hd / 2)): dq and dk leave through the inverse rotary embedding, i.e. they are the
    gradients of the un-rotated projections when q and k were rotated after the projection."""
    b, sq, h, hd = q.shape
    sk, hkv = k.shape[1], k.shape[2]
    if dout.stride(-1) != 1 or dout.stride(2) != hd or (b > 1 and dout.stride(0) != sq * dout.stride(1)):
        dout = dout.contiguous()
    dq = torch.empty((b, sq, h, hd), dtype=q.dtype, device=q.device) if dq is None else dq
    dk = torch.empty((b, sk, hkv, hd), dtype=q.dtype, device=q.device) if dk is None else dk
    dv = torch.empty((b, sk, hkv, hd), dtype=q.dtype, device=q.device) if dv is None else dv
    for t in (dq, dk, dv, out, dout):
        assert _attn_rows_ok(t), "attention gradients need evenly pitched rows with adjacent heads"
    dsum = torch.empty((b, h, sq), dtype=torch.float32, device=q.device)
    dq_acc = torch.empty(attn_bwd_dq_floats(b, sq, sk, h, hd), dtype=torch.float32, device=q.device)
    doc = rng = None
    if doc_ids is not None:
        doc, rng = doc_ids if isinstance(doc_ids, tuple) else doc_blocks(doc_ids, k)
    cos = sin = None
    if rope is not None:
        cos, sin = rope
        assert sq == sk and rope_tables_ok(cos, sin)
        assert cos.shape[-1] == hd // 2 and cos.numel() >= sq * (hd // 2)
    _check(
        lib().kf_attn_bwd_rope_bf16(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), dout.data_ptr(),
                                    lse.data_ptr(), dsum.data_ptr(), dq_acc.data_ptr(), dq.data_ptr(), dk.data_ptr(),
                                    dv.data_ptr(), doc.data_ptr() if doc is not None else None, b, sq, sk, h, hkv, hd,
                                    q.stride(1), k.stride(1), v.stride(1), out.stride(1), dout.stride(1), dq.stride(1),
                                    dk.stride(1), dv.stride(1), float(scale), int(causal),
                                    cos.data_ptr() if cos is not None else None,
                                    sin.data_ptr() if sin is not None else None, _ptr(rng), _stream()),
        "kf_attn_bwd_rope_bf16",
    )
    return dq, dk, dv


# --------------------------------------------------------------------------- fused communication kernels
SYMM_RS_BLOCKS = int(os.environ.get("KF_SYMM_RS_BLOCKS", "296"))        # grid cap of the fused reduce-scatter kernel
SYMM_ADAMW_BLOCKS = int(os.environ.get("KF_SYMM_ADAMW_BLOCKS", "592"))  # grid cap of the fused AdamW + publication kernel


def symm_rs_norm(buf, lo: int, n: int, sumsq_out: torch.Tensor, accumulate: bool, max_blocks: int | None = None) -> None:
    """Average this rank's shard [lo, lo+n) of a symmetric gradient buffer over all ranks (in place, own copy)
    and add the squared norm of the result to ``sumsq_out[0]``.  The kernel runs beside the backward GEMMs on a side
    stream; ``max_blocks`` (default ``KF_SYMM_RS_BLOCKS``) bounds how many SMs it shares with them."""
    max_blocks = SYMM_RS_BLOCKS if max_blocks is None else max_blocks
    partial = torch.empty(1024, dtype=torch.float32, device=buf.tensor.device)
    _check(
        lib().kf_symm_rs_norm_bf16(buf.peer_ptrs, buf.multicast_ptr, buf.world, buf.rank, lo, n, partial.data_ptr(),
                                   sumsq_out.data_ptr(), int(accumulate), max_blocks, _stream()),
        "kf_symm_rs_norm_bf16",
    )


def symm_adamw_bcast(param_buf, grad_shard, m, v, lo: int, n: int, n_decay_global: int, lr, beta1, beta2, eps, wd,
                     step: int, grad_scale=None, skip=None, max_blocks: int | None = None) -> None:
    """AdamW on the shard [lo, lo+n) and store of the new parameters into every rank's parameter buffer."""
    max_blocks = SYMM_ADAMW_BLOCKS if max_blocks is None else max_blocks
    bc1 = 1.0 - beta1**step
    bc2_sqrt = math.sqrt(1.0 - beta2**step)
    _check(
        lib().kf_symm_adamw_bcast_bf16(
            param_buf.peer_ptrs, param_buf.multicast_ptr, param_buf.world, param_buf.rank, grad_shard.data_ptr(),
            m.data_ptr(), v.data_ptr(), lo, n, n_decay_global, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt,
            grad_scale.data_ptr() if grad_scale is not None else None, skip.data_ptr() if skip is not None else None,
            max_blocks, _stream()),
        "kf_symm_adamw_bcast_bf16",
    )


def symm_gather(buf, lo: int, n: int, max_blocks: int = 592) -> None:
    _check(lib().kf_symm_gather_bf16(buf.peer_ptrs, buf.multicast_ptr, buf.world, buf.rank, lo, n, max_blocks, _stream()),
           "kf_symm_gather_bf16")


# --------------------------------------------------------------------------- vocabulary-parallel cross entropy
def ce_vp_stats(logits: torch.Tensor, labels: torch.Tensor, vocab_start: int):
    """Per row of this rank's vocabulary shard (T, V_local) bf16: (max, sum of exp relative to that max, logit of the
    label if the label is in [vocab_start, vocab_start + V_local) else 0), three fp32 (T,) vectors."""
    t, v = logits.shape
    out = torch.empty((3, t), dtype=torch.float32, device=logits.device)
    _check(lib().kf_ce_vp_stats_bf16(logits.data_ptr(), labels.data_ptr(), int(vocab_start), out[0].data_ptr(),
                                     out[1].data_ptr(), out[2].data_ptr(), t, v, logits.stride(0), _stream()),
           "kf_ce_vp_stats_bf16")
    return out[0], out[1], out[2]


def ce_vp_bwd(logits: torch.Tensor, labels: torch.Tensor, vocab_start: int, lse: torch.Tensor, inv_n: torch.Tensor,
              upstream: torch.Tensor | None, z_weight: float) -> torch.Tensor:
    """In place: logits <- gradient of the mean (over valid rows) cross entropy (+ z-loss) given the global
    log-sum-exp ``lse`` (T,); ``inv_n`` and ``upstream`` are device scalars."""
    t, v = logits.shape
    _check(lib().kf_ce_vp_bwd_bf16(logits.data_ptr(), labels.data_ptr(), int(vocab_start), lse.data_ptr(), inv_n.data_ptr(),
                                   upstream.data_ptr() if upstream is not None else None, float(z_weight), t, v,
                                   logits.stride(0), _stream()), "kf_ce_vp_bwd_bf16")
    return logits


# --------------------------------------------------------------------------- sharded parameters (ZeRO-3)
def _ll_array(values):
    return (ctypes.c_longlong * len(values))(*[int(v) for v in values])


def symm_pull(shard_buf, full_offsets, lengths, shard_offsets, dst: torch.Tensor, max_blocks: int = 592) -> None:
    """All-gather of up to 16 parameters of a sharded unit into the full-layout buffer ``dst``: parameter i
    (``lengths[i]`` elements, cut into ``world`` equal pieces) is assembled at ``dst[full_offsets[i]:]`` from every
    rank's piece at ``shard_offsets[i]`` of its shard (``shard_buf``: the symmetric shard buffer)."""
    _check(lib().kf_symm_pull_bf16(shard_buf.peer_ptrs, shard_buf.world, len(lengths), _ll_array(full_offsets),
                                   _ll_array(lengths), _ll_array(shard_offsets), dst.data_ptr(), max_blocks, _stream()),
           "kf_symm_pull_bf16")


def symm_rs_shard(grad_buf, full_offsets, lengths, shard_offsets, shard_grad: torch.Tensor, accumulate: bool,
                  max_blocks: int | None = None) -> None:
    """Reduce-scatter of full-layout gradient staging buffers (``grad_buf``: symmetric) into this rank's gradient
    shard: the mean over ranks of this rank's piece of every listed parameter is written (or added) to
    ``shard_grad[shard_offsets[i]:]``."""
    max_blocks = SYMM_RS_BLOCKS if max_blocks is None else max_blocks
    _check(lib().kf_symm_rs_shard_bf16(grad_buf.peer_ptrs, grad_buf.multicast_ptr, grad_buf.world, grad_buf.rank,
                                       len(lengths), _ll_array(full_offsets), _ll_array(lengths), _ll_array(shard_offsets),
                                       shard_grad.data_ptr(), int(accumulate), max_blocks, _stream()),
           "kf_symm_rs_shard_bf16")


def gemm_gather(x2: torch.Tensor, plan: dict, n: int, *, epi: int = 0, residual: torch.Tensor | None = None,
                rope: tuple | None = None, want_gu: bool = True):
    """GEMM whose weight operand is gathered from the data-parallel ranks' parameter shards inside the kernel.

    ``plan`` comes from ``ShardedDataParallelEngine.gather_plan`` (shard buffer, segment rows / shard offsets, the
    staging view that receives the operand, scratch flags).  ``epi`` 0: ``x W^T (+ residual)`` -> (M, n);
    1: SwiGLU over W = [gate ; up] with hidden size ``n`` -> (h (M, n), gu (M, 2n) or None); 2: rotary epilogue
    (``rope`` as in :func:`gemm`) -> (M, n).  Afterwards the staging view holds the whole weight."""
    m, k = x2.shape
    symm = plan["symm"]
    out = torch.empty((m, n), dtype=torch.bfloat16, device=x2.device)
    r_ptr, ldr, gu = None, 0, None
    if epi == 1 and want_gu:
        gu = torch.empty((m, 2 * n), dtype=torch.bfloat16, device=x2.device)
        r_ptr, ldr = gu.data_ptr(), 2 * n
    elif epi == 0 and residual is not None:
        assert residual.shape == (m, n) and residual.stride(1) == 1
        r_ptr, ldr = residual.data_ptr(), residual.stride(0)
    cos_p = sin_p = None
    s_len = rope_cols = hd = 0
    if epi == 2:
        cos, sin, s_len, rope_cols, hd = rope
        cos_p, sin_p = cos.data_ptr(), sin.data_ptr()
    code = lib().kf_gemm_gather_bf16(
        epi, x2.data_ptr(), out.data_ptr(), r_ptr, m, n, k, x2.stride(0), n, ldr, symm.peer_ptrs, symm.world, symm.rank,
        len(plan["seg_rows"]), _ll_array(plan["seg_rows"]), _ll_array(plan["seg_src"]), plan["stage"].data_ptr(),
        plan["flags"].data_ptr(), cos_p, sin_p, int(s_len), int(rope_cols), int(hd), sm_count(), _stream())
    _check(code, "kf_gemm_gather_bf16")
    return (out, gu) if epi == 1 else out
