"""A transformer block without gradients (generation, evaluation) on the native kernels.

One new token per sequence against a KV cache runs as one native call that issues the whole chain (``kf_block_decode_bf16``:
RMSNorm, q|k|v projection with the rotary embedding written straight into the cache, split attention over the cache,
o projection with the residual, RMSNorm, gate|up with SwiGLU, down with the residual).  A prompt that starts an empty cache,
or a plain forward pass, uses the epilogue-fused GEMMs of the training block and reads q | k | v from the projection's own
buffer.  The weights of separate ``nn.Linear`` modules are read where they are: nothing is concatenated.

All blocks of a model on one new token are one native call (:func:`run_layers`).  A step through plain blocks is checked in
native code too (``csrc/steps.cpp``), by the rules of :func:`_plan`, which decides about every other call.

What the fused form does not cover (masks, hooks, q/k norms, tensor parallelism, fp8, captured attention weights, a prompt
behind a non-empty cache, foreign module types) returns None and takes the op-by-op path.

Semantics: kempnerforge/model/transformer.py:82-103, kempnerforge/model/attention.py:116-236.
"""

from __future__ import annotations

import math

import torch
from torch.nn.modules import module as _nn_module

from kempnerforge_b200.models.attention import Attention, KVCache
from kempnerforge_b200.models.mlp import SwiGLUMLP
from kempnerforge_b200.models.norm import RMSNorm
from kempnerforge_b200.ops import cuda as kc
from kempnerforge_b200.ops import functional as F

_BF16 = torch.bfloat16


def _plain(mod) -> bool:
    """No hooks and no replaced ``forward``: calling the module does nothing but its class's own forward."""
    return not (mod._forward_hooks or mod._forward_pre_hooks or "forward" in mod.__dict__)


def _weight(mod, name: str):
    """``mod.name.weight`` straight from the module tables (None when it is not a plain parameter there): a generation step
    reads seven of them per block, and ``Module.__getattr__`` costs more than the checks that follow."""
    sub = mod._modules.get(name)
    return None if sub is None else sub._parameters.get("weight")


def _matrix(w, rows: int, cols: int) -> int:
    """Device address of a dense, 16-byte aligned bf16 (rows, cols) matrix on a GPU; 0 for anything else."""
    if (w is None or w.dtype is not _BF16 or not w.is_cuda or w.dim() != 2 or w.size(0) != rows or w.size(1) != cols
            or not w.is_contiguous() or hasattr(w, "_kf_fp8")):
        return 0
    p = w.data_ptr()
    return 0 if p & 15 else p


def _gain(norm, d: int) -> int:
    """Device address of a plain RMSNorm's bf16 gain of width d; 0 for any other norm."""
    if type(norm) is not RMSNorm or not _plain(norm):
        return 0
    w = norm._parameters.get("weight")
    if w is None or w.dtype is not _BF16 or not w.is_cuda or w.dim() != 1 or w.size(0) != d or not w.is_contiguous():
        return 0
    p = w.data_ptr()
    return 0 if p & 15 else p


class _Plan:
    """Addresses and sizes of one block's weights and cache, checked."""

    __slots__ = ("mlp", "norm1", "norm2", "attn_ptrs", "mlp_ptrs", "cache_ptrs", "weights", "h", "hkv", "hd", "f", "past", "batch_step",
                 "eps1", "eps2")


def _plan(block, b: int, s: int, d: int, cos, sin, cache):
    """The plan of a call of ``block`` on (b, s, d) inputs, or None when this path does not cover it."""
    sub = block._modules
    att, mlp, norm1 = sub["attention"], sub["mlp"], sub["attention_norm"]
    if (type(att) is not Attention or att.tp is not None or att._modules.get("q_norm") is not None or att.q_norm is not None
            or att.k_norm is not None or att.capture_attention_weights or getattr(block, "fp8", False)
            or getattr(block, "_kf_fp8_block", False) or not _plain(att)):
        return None
    p = _Plan()
    hd = p.hd = att.head_dim
    wq, wk, wv, wo = _weight(att, "q_proj"), _weight(att, "k_proj"), _weight(att, "v_proj"), _weight(att, "o_proj")
    if hd not in (64, 128) or b * s == 0 or d % 8 or wq is None or wk is None:
        return None
    qc, kvc = wq.size(0), wk.size(0)
    if kvc == 0 or qc % hd or kvc % hd or qc % kvc or getattr(getattr(wq, "_kf_flat", None), "sharded", False):
        return None
    p.attn_ptrs = _gain(norm1, d), _matrix(wq, qc, d), _matrix(wk, kvc, d), _matrix(wv, kvc, d), _matrix(wo, d, qc)
    if (not all(p.attn_ptrs) or cos.dtype is not torch.float32 or sin.dtype is not torch.float32 or cos.dim() != 2
            or cos.shape != sin.shape or cos.size(0) < s or cos.size(1) != hd // 2
            or not (cos.is_cuda and cos.is_contiguous() and sin.is_contiguous())):
        return None
    p.h, p.hkv, p.past = qc // hd, kvc // hd, 0
    if cache is not None:
        k, v = cache.k, cache.v
        p.past = cache.seq_len
        if (type(cache) is not KVCache or k.dtype is not _BF16 or v.dtype is not _BF16 or k.dim() != 4 or k.shape != v.shape
                or k.size(0) != b or k.size(2) != p.hkv or k.size(3) != hd or not (k.is_contiguous() and v.is_contiguous())
                or not (k.is_cuda and v.is_cuda) or p.past + s > k.size(1)):
            return None
        p.cache_ptrs, p.batch_step = (k.data_ptr(), v.data_ptr()), k.stride(0)
        if (p.cache_ptrs[0] | p.cache_ptrs[1]) & 15:
            return None
    p.mlp_ptrs, p.norm2, p.f, p.eps1, p.eps2 = None, None, 0, norm1.eps, 0.0
    wg = wu = wd = None
    if type(mlp) is SwiGLUMLP and mlp.tp is None and _plain(mlp):
        norm2 = sub["mlp_norm"]
        wg, wu, wd = _weight(mlp, "gate_proj"), _weight(mlp, "up_proj"), _weight(mlp, "down_proj")
        f = wg.size(0) if wg is not None else 0
        ptrs = _matrix(wg, f, d), _matrix(wu, f, d), _matrix(wd, d, f)
        g2 = _gain(norm2, d) if f and f % 8 == 0 and all(ptrs) else 0
        if g2:
            p.mlp_ptrs, p.norm2, p.f, p.eps2 = (g2, *ptrs), norm2, f, norm2.eps
    p.mlp, p.norm1, p.weights = mlp, norm1, (wq, wk, wv, wo, wg, wu, wd)
    return p


def _refused() -> bool:
    return bool(_nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks
                or torch.autograd.forward_ad._current_level >= 0 or kc.attn_policy() != "native")


def _one_token(b: int, cos, sin) -> bool:
    """The native generation step takes this many sequences and these tables."""
    return b <= kc.SKINNY_MAX_ROWS and not (cos.data_ptr() | sin.data_ptr()) & 15


def run_layers(layers, x, cos, sin, caches):
    """One new token per sequence through all of a model's blocks as one native call, checks included: the last block's output
    (B, 1, D), or None when some block is not plainly covered (nothing has been done then).  Issued block by block, Python takes
    50 us per block, more than the 18 us that the five kernels of a small one run."""
    if x.dim() != 3 or x.size(1) != 1 or not layers or len(caches) < len(layers) or _refused():
        return None
    return kc.blocks_decode(list(layers), list(caches), x if x.is_contiguous() else x.contiguous(), cos, sin)


def run(block, x, cos, sin, cache):
    """The block's output (new (B, S, D) tensor), or None when this path does not cover the call."""
    if x.dim() != 3 or _refused():
        return None
    b, s, d = x.shape
    if s == 1 and type(cache) is KVCache:   # a generation step of a plain block is checked and issued by one native call
        def foreign(q2, h, hd, past):
            out = F.attention(q2.unflatten(1, (h, hd)).unsqueeze(1), cache.k[:, : past + 1], cache.v[:, : past + 1], causal=False)
            return out.reshape(b, h * hd)   # SDPA's output is a transposed view

        y = kc.blocks_decode([block], [cache], x if x.is_contiguous() else x.contiguous(), cos, sin, foreign)
        if y is not None:
            return y
    p = _plan(block, b, s, d, cos, sin, cache)
    if p is None:
        return None
    hd, h, hkv, past, g2, norm1, norm2 = p.hd, p.h, p.hkv, p.past, p.mlp_ptrs, p.norm1, p.norm2
    wq, wk, wv, wo, wg, wu, wd = p.weights
    mlp, qc = p.mlp, h * hd
    if not x.is_contiguous():
        x = x.contiguous()
    xp = x.data_ptr()
    if xp & 15:
        return None
    scale = 1.0 / math.sqrt(hd)
    t = b * s
    if s == 1 and cache is not None:
        if not _one_token(b, cos, sin):
            return None
        y = torch.empty((b, 1, d), dtype=_BF16, device=x.device)

        kc.block_decode(y, (xp, *p.attn_ptrs), p.mlp_ptrs, p.cache_ptrs, (cos.data_ptr(), sin.data_ptr()),
                        (b, d, h, hkv, hd, p.f, past, p.batch_step), (p.eps1, p.eps2, scale),
                        lambda q2: foreign(q2, h, hd, past))
        cache.seq_len = past + 1
        return y if g2 else y + mlp(block.mlp_norm(y))
    if past:
        return None
    x2 = x.view(t, d)
    n1, _ = kc.rmsnorm_fwd(x2, norm1.weight, norm1.eps)
    qkv = kc.qkv_rope(n1, [wq, wk, wv], cos, sin, s, hd)
    qkv4 = qkv.view(b, s, h + 2 * hkv, hd)
    q, k_new, v_new = qkv4[:, :, :h], qkv4[:, :, h : h + hkv], qkv4[:, :, h + hkv :]
    if cache is not None:   # empty so far, and one that the plan has checked
        if cache.k.device == cache.v.device == x.device and 2 * t * hkv * hd < 1 << 31:
            kc.cache_rows(qkv[:, qc:], cache.k, cache.v, s)
            cache.seq_len = s
        else:
            cache.update(k_new, v_new)
    attn, _ = kc.attn_fwd(q, k_new, v_new, True, None, scale)
    h1 = kc.gemm_rows(attn.view(t, qc), [wo], residual=x2)
    if not g2:
        y = h1.view(b, s, d)
        return y + mlp(block.mlp_norm(y))
    n2, _ = kc.rmsnorm_fwd(h1, norm2.weight, norm2.eps)
    hid = kc.swiglu_rows(n2, wg, wu)
    return kc.gemm_rows(hid, [wd], residual=h1).view(b, s, d)
