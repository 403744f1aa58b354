"""Autograd wrappers of the native mixture-of-experts kernels: fused router, stable sort by expert, row gather and
weighted combine.  Every piece stays on the device and has a native backward.

Parity: kempnerforge/model/router.py:45-72,157-200 and kempnerforge/model/moe.py:256-349 (same mathematics: softmax
or sigmoid(+bias) scores, top-k, renormalised weights, Switch load-balancing loss E * sum(f_e * P_e), z-loss
mean(logsumexp²), sort by expert, weighted sum over the k expert outputs).
"""

from __future__ import annotations

import torch

from kempnerforge_b200.ops import cuda as kc


def native_ok(x: torch.Tensor, num_experts: int, top_k: int) -> bool:
    from kempnerforge_b200.ops import functional as F

    if F._FORCE_REF:
        return False
    return (x.is_cuda and kc.available() and getattr(kc.lib(), "kf_router_topk", None) is not None
            and num_experts <= 256 and top_k <= 8 and top_k <= num_experts)


class _RouterFn(torch.autograd.Function):
    """(weights, indices, counts, score_mean, z_loss, balance) from logits; weights in ``dtype``.  ``score_mean`` (mean score per
    expert), ``z_loss`` and, for softmax scores, ``balance`` = E sum(counts / (T k) * score_mean) are differentiable, like
    ``weights``; ``indices`` and ``counts`` are not."""

    @staticmethod
    def forward(ctx, logits, bias, sigmoid, k, dtype):
        ctx.set_materialize_grads(False)   # a layer that trains on the weights alone gets None for the rest
        logits = logits.contiguous()
        b = bias
        if b is not None:
            b = b.detach()
            if b.dtype not in (torch.float32, torch.bfloat16):
                b = b.to(torch.float32)
            b = b.contiguous()
        # the sigmoid router nudges its bias in place right after routing: the fp32 copy in ``keep`` serves the backward
        w, w16, idx, keep, counts, mean, z, balance = kc.router_topk(logits, b, sigmoid, k, dtype is torch.bfloat16)
        ctx.save_for_backward(logits, idx, w, keep)
        ctx.sigmoid, ctx.has_bias = sigmoid, bias is not None
        ctx.bias_dtype = bias.dtype if bias is not None else None
        ctx.mark_non_differentiable(idx, counts, *((balance,) if sigmoid else ()))
        out = w16 if dtype is torch.bfloat16 else w.to(dtype)
        return out, idx, counts, mean, z, balance

    @staticmethod
    def backward(ctx, dw, _didx, _dcounts, dmean, dz, dbalance):
        logits, idx, w, keep = ctx.saved_tensors   # keep: the bias (sigmoid) or the counts (softmax)
        t, e = logits.shape
        if dw is None and dmean is None and dz is None and dbalance is None:
            return None, None, None, None, None
        dmean, dz, dbalance = (None if g is None else g.float().contiguous() for g in (dmean, dz, dbalance))
        if not torch.is_grad_enabled():
            if dw is not None:
                dw = (dw if dw.dtype in (torch.float32, torch.bfloat16) else dw.float()).contiguous()
            bias_grad = ctx.bias_dtype if ctx.has_bias and ctx.needs_input_grad[1] else None
            half = bias_grad is torch.bfloat16
            dlogits, dbias = kc.router_bwd(logits, keep, ctx.sigmoid, idx, w, dw, dmean, dz, dbalance,
                                           None if bias_grad is None else torch.bfloat16 if half else torch.float32)
            return dlogits, dbias.to(bias_grad) if dbias is not None else None, None, None, None
        # create_graph: the same formulas as differentiable element-wise ops
        lf = logits.float()
        if ctx.sigmoid:
            scores = torch.sigmoid(lf + keep)
        else:
            scores = torch.softmax(lf, dim=-1)
        dscores = torch.zeros_like(scores)
        if dw is not None:
            sel = scores.gather(1, idx)
            ssum = sel.sum(dim=1, keepdim=True)
            # w = sel / ssum
            dw = dw.float()
            dsel = (dw - (dw * (sel / ssum)).sum(dim=1, keepdim=True)) / ssum
            dscores = dscores.scatter(1, idx, dsel)
        if dbalance is not None:
            per_expert = dbalance * e * keep / (t * idx.shape[1])
            dmean = per_expert if dmean is None else dmean + per_expert
        if dmean is not None:
            dscores = dscores + dmean[None, :] / t
        if ctx.sigmoid:
            dlogits = dscores * scores * (1.0 - scores)
        else:
            dlogits = scores * (dscores - (dscores * scores).sum(dim=1, keepdim=True))
        if dz is not None:
            lse = torch.logsumexp(lf, dim=-1, keepdim=True)
            dlogits = dlogits + (dz * 2.0 / t) * lse * torch.softmax(lf, dim=-1)
        # expert_bias is nudged by its own rule, never by gradients through the scores (the reference detaches
        # nothing here either, but its bias update overwrites any gradient step); keep autograd's answer
        dbias = dlogits.sum(dim=0).to(ctx.bias_dtype) if (ctx.has_bias and ctx.needs_input_grad[1]) else None
        return dlogits.to(logits.dtype), dbias, None, None, None


def route(logits: torch.Tensor, bias: torch.Tensor | None, sigmoid: bool, k: int):
    """(weights fp32, indices, counts, score_mean, z_loss)."""
    return _RouterFn.apply(logits, bias, sigmoid, k, torch.float32)[:5]


def route_layer(logits: torch.Tensor, bias: torch.Tensor | None, sigmoid: bool, k: int, dtype: torch.dtype):
    """(weights in ``dtype``, indices, counts, score_mean, z_loss, balance) of :class:`_RouterFn`."""
    return _RouterFn.apply(logits, bias, sigmoid, k, dtype)


class _GatherFn(torch.autograd.Function):
    """x_sorted[row] = x[token of row]; backward sums the k rows of every token."""

    @staticmethod
    def forward(ctx, x, slot_of_row, row_of_slot, k):
        ctx.save_for_backward(row_of_slot)
        ctx.k, ctx.tokens = k, x.shape[0]
        return kc.moe_gather(x.contiguous(), slot_of_row, k)

    @staticmethod
    def backward(ctx, dy):
        (row_of_slot,) = ctx.saved_tensors
        return kc.moe_combine(dy.contiguous(), row_of_slot, None, ctx.tokens, ctx.k), None, None, None


class _CombineFn(torch.autograd.Function):
    """out[t] = sum_j w[t, j] * y_sorted[row_of_slot[t, j]] (+ plus[t])."""

    @staticmethod
    def forward(ctx, y, w, row_of_slot, slot_of_row, plus):
        t, k = w.shape
        wk = (w if w.dtype in (torch.float32, torch.bfloat16) else w.float()).contiguous()
        ctx.save_for_backward(y, wk, row_of_slot, slot_of_row)
        ctx.w_dtype = w.dtype
        return kc.moe_combine(y.contiguous(), row_of_slot, wk, t, k, plus)

    @staticmethod
    def backward(ctx, dout):
        y, wk, row_of_slot, slot_of_row = ctx.saved_tensors
        t, k = wk.shape
        dy, dw_rows = kc.moe_combine_bwd(dout.contiguous(), y.contiguous(), slot_of_row, wk.reshape(-1), k)
        # dw comes out per sorted row (indexed by slot inside the kernel): it is already in slot order
        return dy, dw_rows.view(t, k).to(ctx.w_dtype), None, None, dout if ctx.needs_input_grad[4] else None


def sort_by_expert(indices: torch.Tensor, num_experts: int):
    return kc.moe_sort(indices.contiguous(), num_experts)


def gather_rows(x, slot_of_row, row_of_slot, k):
    return _GatherFn.apply(x, slot_of_row, row_of_slot, k)


def combine_rows(y, w, row_of_slot, slot_of_row, plus=None):
    """``plus`` (T, D): another contribution to every token (a shared expert), added to the rounded sum in the same pass."""
    if plus is not None and not (plus.is_cuda and plus.dtype == y.dtype and plus.shape == (w.shape[0], y.shape[1])
                                 and plus.is_contiguous() and plus.data_ptr() % 16 == 0):
        return _CombineFn.apply(y, w, row_of_slot, slot_of_row, None) + plus
    return _CombineFn.apply(y, w, row_of_slot, slot_of_row, plus)
