"""`torch.autograd.Function`s with the interface of the reference's
``flashlinear.LinearAttention`` (flashlinear/linear_attn.py:11-31) and
``flashlinear.LinearAttentionSmallVHD`` (flashlinear/linear_attn_smallv_hd.py:14-36):
``.apply(q, k, v)`` returns the unnormalised causal ``(Q K^T (.) M) V`` in bf16, saves q, k, v (plus
the small fp32 final state when the backward can use it) and returns three bf16 gradients from
backward. Under autocast the inputs are cast to bf16 exactly as
the reference's ``custom_fwd(cast_inputs=torch.bfloat16)`` does.
"""
from __future__ import annotations

import functools
from typing import Any, Tuple

import torch
from torch.autograd import Function

from . import ops


def _autocast_to_bf16(forward):
    """``custom_fwd(cast_inputs=torch.bfloat16)``, entered only where autocast is on. The backward
    needs no counterpart: nothing it calls depends on the autocast state."""
    cast = torch.amp.custom_fwd(device_type="cuda", cast_inputs=torch.bfloat16)(forward)

    @functools.wraps(forward)
    def wrapper(ctx: Any, *args):
        return cast(ctx, *args) if torch.is_autocast_enabled("cuda") else forward(ctx, *args)

    return wrapper


def _forward_with_state(ctx: Any, q, k, v, smallv: bool):
    """Forward through the reference-named wrapper's checks; when a backward will follow and can
    use it, also keeps the final state S = sum k^T v (fp32, batch*heads x dk x dv), which lets the
    backward read q, k, v, dO from HBM once instead of twice, and with few heads per GPU the states
    at the boundaries of the forward's segments."""
    ops.check_forward_preconditions(q, v, smallv)
    need_grad = any(ctx.needs_input_grad[:3])
    ctx.keep_padded = False
    if smallv and need_grad and q.is_cuda and q.shape[-1] % 8 != 0:
        # Head dims such as 273 have rows the kernels cannot address in place. Repack q and k once,
        # keep the repacked views for the backward, and let the backward return dQ and dK as views
        # of row-padded tensors (same values and shape as the reference's gradients, which are
        # contiguous, linear_attn_kernels_smallv_hd.py:384-386; one copy pass per tensor less).
        q, k = ops.kernel_view(q), ops.kernel_view(k)
        ctx.keep_padded = True
    res = ops.host_forward(q, k, v, None, 2 if need_grad else 0)
    if res is None:
        res = ops.general_forward(q, k, v) if need_grad else (ops.causal_dot_product_fwd(q, k, v), None, None, None)
    out, s_final, seg_states, views = res
    # Head dims whose rows had to be repacked: the backward reads the repacked copies again (a pad
    # pass over three tensors less). They are kept in place of q, k, v, not beside them; what is left of
    # those is their layout, which the gradients take, and their version counts.
    ctx.strides, versions = None, ()
    if views is not None:
        ctx.strides, versions = [t.stride() for t in (q, k, v)], ops.versions_of(q, k, v)
        q, k, v = views
    ctx.save_for_backward(q, k, v, s_final, seg_states, *versions)
    return out


def _backward_with_state(ctx: Any, grad_output):
    q, k, v, s_final, seg_states = ctx.saved_tensors[:5]
    if ctx.strides is not None:
        res = ops.host_backward(grad_output, q, k, v, s_last=s_final, seg_states=seg_states,
                                keep_padded=ctx.keep_padded, strides=ctx.strides)
        if res is not None:
            return res
    return ops.causal_dot_product_bwd(grad_output, q, k, v, s_last=s_final, seg_states=seg_states,
                                      keep_padded=ctx.keep_padded)


class LinearAttention(Function):
    """Causal linear attention with dk == dv."""

    @staticmethod
    @_autocast_to_bf16
    def forward(ctx: Any, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
        return _forward_with_state(ctx, q, k, v, smallv=False)

    @staticmethod
    def backward(ctx: Any, grad_output: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
        return _backward_with_state(ctx, grad_output)


class LinearAttentionSmallVHD(Function):
    """Causal linear attention where q/k have head dim hd_qk and v has a smaller hd_v."""

    @staticmethod
    @_autocast_to_bf16
    def forward(ctx: Any, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
        return _forward_with_state(ctx, q, k, v, smallv=True)

    @staticmethod
    def backward(ctx: Any, grad_output: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
        return _backward_with_state(ctx, grad_output)


class LinearAttentionResumable(Function):
    """Causal linear attention that carries its running state across calls.

    ``out, s_final = LinearAttentionResumable.apply(q, k, v, s_init)`` where ``s_init`` /
    ``s_final`` are fp32 ``[batch, heads, dk, dv]`` (sum of k_j^T v_j over the tokens before /
    up to the end of this call; ``s_init=None`` starts from zero). Feeding ``s_final`` of one call
    as ``s_init`` of the next gives what one call over the concatenated tokens gives: chunked
    prefill, decoding a few tokens at a time, or training on a long sequence piece by piece. Any
    number of tokens per call is accepted (the reference's multiple-of-64 rule,
    linear_attn_kernels.py:323-325, is a property of its tiling; calls of up to 16 tokens, 8
    where both head dims are at most 64, run the recurrence itself in fp32 instead of a 128-token tile). The state is
    differentiable: the backward returns the gradient of ``s_init`` and accepts one for ``s_final``.

    Not part of the reference, whose Functions (flashlinear/linear_attn.py:11-31) always start from
    an empty state. Head dims up to 128.
    """

    @staticmethod
    @_autocast_to_bf16
    def forward(ctx: Any, q, k, v, s_init=None):
        assert q.shape[-1] <= ops.KERNEL_HEAD_DIM and v.shape[-1] <= ops.KERNEL_HEAD_DIM, \
            f"Only head_dims <= {ops.KERNEL_HEAD_DIM} are supported."
        B, H, _, dk = q.shape
        dv = v.shape[-1]
        if s_init is not None:
            # autocast's cast_inputs also turns the fp32 state to bf16; the state stays fp32
            s_init = s_init.to(torch.float32).contiguous()
            if tuple(s_init.shape) != (B, H, dk, dv):
                raise ValueError(f"s_init must have shape {(B, H, dk, dv)}")
        flat_init = None if s_init is None else s_init.view(B * H, dk, dv)
        res = ops.host_forward(q, k, v, flat_init, 1)
        if res is not None:
            out, s_final = res[:2]
        else:
            s_final = torch.empty(B, H, dk, dv, dtype=torch.float32, device=q.device)
            out = ops.causal_dot_product_fwd(q, k, v, s_init=flat_init, s_final=s_final.view(B * H, dk, dv))
        ctx.save_for_backward(q, k, v, s_init, s_final)
        return out, s_final

    @staticmethod
    def backward(ctx: Any, grad_output, grad_s_final):
        q, k, v, s_init, s_final = ctx.saved_tensors
        B, H, _, dk = q.shape
        dv = v.shape[-1]
        flat = (B * H, dk, dv)
        if grad_output is None:
            grad_output = torch.zeros_like(v)
        r_init = None if grad_s_final is None else grad_s_final.to(torch.float32).contiguous().view(flat)
        r_final = torch.empty(flat, dtype=torch.float32, device=q.device) if ctx.needs_input_grad[3] else None
        s_last = s_final.view(flat) if ops.backward_uses_final_state(q, v) else None
        dq, dk_, dv_ = ops.causal_dot_product_bwd(
            grad_output.contiguous(), q, k, v,
            s_init=None if s_init is None else s_init.view(flat),
            r_init=r_init, r_final=r_final, s_last=s_last)
        return dq, dk_, dv_, None if r_final is None else r_final.view(B, H, dk, dv)


class LinearAttentionNormalized(Function):
    """Causal linear attention WITH its denominator:
    ``out_i = sum_{j<=i} (q_i . k_j) v_j / (q_i . sum_{j<=i} k_j + eps)``, i.e. the whole recipe of
    the reference's README (README.md:27-30) in one Function. The product runs in the same kernels
    as LinearAttention / LinearAttentionSmallVHD. The denominator and the division run inside the
    forward product where ``ops.normalized_fused`` says so (bf16, dk == dv <= 128, enough heads),
    otherwise, like their gradients, in streaming kernels with an fp32 running sum instead of
    PyTorch's cumsum / multiply / sum / divide passes. ``apply(q, k, v, eps=1e-5)``; dv a multiple of 8.
    """

    @staticmethod
    @_autocast_to_bf16
    def forward(ctx: Any, q, k, v, eps: float = 1e-5):
        ops.check_forward_preconditions(q, v, smallv=q.shape[-1] != v.shape[-1])
        if v.shape[-1] % 8 != 0:
            raise NotImplementedError("LinearAttentionNormalized needs a value head dim that is a multiple of 8")
        q, k = ops.kernel_view(q), ops.kernel_view(k)  # repacked once if the rows are not 16-byte multiples
        B, H, _, dk = q.shape
        need_grad = any(ctx.needs_input_grad[:3])
        if ops.normalized_fused(q, k, v):
            out, den, s_final = ops.normalized_fwd(q, k, v, eps, need_grad)
            ctx.has_state = s_final is not None
            ctx.save_for_backward(q, k, v, out, den, *((s_final,) if ctx.has_state else ()))
            return out
        s_final = None
        if need_grad and ops.backward_uses_final_state(q, v):
            s_final = torch.empty(B * H, dk, v.shape[-1], dtype=torch.float32, device=q.device)
        out = ops.causal_dot_product_fwd(q, k, v, s_final=s_final)
        if not out.is_contiguous():
            out = out.contiguous()
        den = ops.normalize_fwd(q, k, out, eps)
        ctx.has_state = s_final is not None
        if ctx.has_state:
            ctx.save_for_backward(q, k, v, out, den, s_final)
        else:
            ctx.save_for_backward(q, k, v, out, den)
        return out

    @staticmethod
    def backward(ctx: Any, grad_output):
        saved = ctx.saved_tensors
        q, k, v, out, den = saved[:5]
        s_final = saved[5] if ctx.has_state else None
        dnum, dden = ops.normalize_bwd_prepare(grad_output, out, den)
        grads = ops.normalized_bwd(dnum, dden, q, k, v, s_final)
        if grads is not None:
            return grads + (None,)
        dq, dk, dv = ops.causal_dot_product_bwd(dnum, q, k, v, s_last=s_final, keep_padded=True)
        ops.normalize_bwd_sweep(q, k, dq, dk, dden)
        return dq, dk, dv, None


class TaylorLinearAttention(Function):
    """Causal linear attention on second-order Taylor features of RAW q, k:
    ``apply(xq, xk, v)`` with xq, xk ``[B, H, N, d]`` (d = 8 or 16) and v ``[B, H, N, dv]`` (dv <= 64)
    returns ``sum_{j<=i} (phi(xq_i) . phi(xk_j)) v_j`` with ``phi(x) = [1, x / d^(1/4),
    vec(x x^T) / (sqrt(2) sqrt(d))]`` (benchmark configuration 4: d = 16 -> 273 features), and its
    backward returns gradients with respect to the raw xq, xk and v.

    With values of 8, 16, 32 or 64 columns the features are formed on chip and never exist in memory, in neither
    pass, and nothing but xq, xk and v is kept for the backward. Other powers of two go through feature tensors in memory,
    which are kept, and so do few heads with many tokens at d = 8, where that is faster (see
    ``ops._taylor_memory_is_faster``); widths that are no power of two are refused (as by ``LinearAttentionSmallVHD``).
    The reference has no counterpart.
    """

    @staticmethod
    @_autocast_to_bf16
    def forward(ctx: Any, xq, xk, v):
        out, features = ops.taylor_forward(xq, xk, v), ()
        if out is None:  # errors, and what does not run on chip
            out, *features = ops.taylor_forward_in_memory(xq, xk, v)
            if ops._taylor_on_chip(xq, xk, v, backward=True):
                features = ()
        ctx.save_for_backward(xq, xk, v, *features)
        return out

    @staticmethod
    def backward(ctx: Any, grad_output):
        xq, xk, v, *features = ctx.saved_tensors
        if not features:
            grads = ops.taylor_backward(grad_output, xq, xk, v)
            if grads is not None:
                return tuple(grads)
            features = ops.taylor_features(xq), ops.taylor_features(xk)
        return ops.taylor_backward_in_memory(grad_output, xq, xk, v, *features)
