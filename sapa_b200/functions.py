"""Operators of SAPA-B: ``qk`` (sim), ``av`` (atn), the fused ``sapa_fused`` and its channels-last form.

``qk`` and ``av`` keep the names, positional arguments, assertions and error behaviour of the reference's
``QKFunction`` / ``AVFunction`` (sapa/sapa/sapa_func.py:9-96): AssertionError on inconsistent shapes,
NotImplementedError for CPU tensors, RuntimeError for non-contiguous tensors, ``None`` gradients for the
two integers.  Checks, allocation and the autograd nodes are native (``csrc/host.cpp``): the Python layer of a call is one
function call.  The ``Function`` classes run the same native code for traces and transforms (``_lib.transformed``), and for
callers who use them by name.
"""
from __future__ import annotations

import torch
from torch.autograd import Function

from . import _lib


def qk(query, key, kernel_size, scale_factor):
    """Local similarity: out[n, dy*K+dx, ph, pw] = <query[n,:,ph,pw], key[n,:,ph/s-r+dy, pw/s-r+dx]>."""
    if _lib.transformed():
        return QKFunction.apply(query, key, kernel_size, scale_factor)
    return (_lib.host or _lib.load_host()).qk(query, key, kernel_size, scale_factor)


def av(attn, value, kernel_size, scale_factor):
    """Aggregation: out[n, c, ph, pw] = sum_k attn[n, k, ph, pw] * value[n, c, window_k(ph, pw)]."""
    if _lib.transformed():
        return AVFunction.apply(attn, value, kernel_size, scale_factor)
    return (_lib.host or _lib.load_host()).av(attn, value, kernel_size, scale_factor)


def sapa_fused(query, key, value, kernel_size=5, scale_factor=2):
    """atn(softmax(sim(query, key)), value) as one op (the whole of ``SAPA.attention``, sapa_base.py:38-40);
    differentiable with respect to query, key and value.

    With a fused kernel available the attention map stays in registers (it is written once, for the backward
    pass, only when a gradient is required); otherwise the three separate kernels run."""
    if _lib.transformed():
        return SapaFusedFunction.apply(query, key, value, kernel_size, scale_factor)
    return (_lib.host or _lib.load_host()).sapa_fused(query, key, value, kernel_size, scale_factor)


class QKFunction(Function):
    """``qk`` under the name that the reference exposes."""

    @staticmethod
    def forward(ctx, query, key, kernel_size, scale_factor):
        ctx.window = (kernel_size, scale_factor)
        ctx.save_for_backward(query, key)
        return _lib.load_host().qk(query, key, kernel_size, scale_factor)

    @staticmethod
    def backward(ctx, grad_output):
        return (*_lib.load_host().qk_backward(grad_output, *ctx.saved_tensors, *ctx.window), None, None)


class AVFunction(Function):
    """``av`` under the name that the reference exposes."""

    @staticmethod
    def forward(ctx, attn, value, kernel_size, scale_factor):
        ctx.window = (kernel_size, scale_factor)
        ctx.save_for_backward(attn, value)
        return _lib.load_host().av(attn, value, kernel_size, scale_factor)

    @staticmethod
    def backward(ctx, grad_output):
        return (*_lib.load_host().av_backward(grad_output, *ctx.saved_tensors, *ctx.window), None, None)


class SapaFusedFunction(Function):
    @staticmethod
    def forward(ctx, query, key, value, kernel_size, scale_factor):
        ctx.window = (kernel_size, scale_factor)
        out, attn = _lib.load_host().sapa_fused_forward(query, key, value, kernel_size, scale_factor, any(ctx.needs_input_grad[:3]))
        if attn is not None:
            ctx.save_for_backward(query, key, value, attn)
        return out

    @staticmethod
    def backward(ctx, grad_output):
        return (*_lib.load_host().sapa_fused_backward(grad_output, *ctx.saved_tensors, *ctx.window), None, None)


def fused_supported(kernel_size: int, scale_factor: int, dtype: torch.dtype) -> bool:
    """True when ``sapa_fused_forward`` has a single-kernel implementation for this configuration."""
    return scale_factor == 2 and kernel_size in (3, 5) and dtype in (torch.float32, torch.float16, torch.bfloat16)


def fused_forward_raw(query, key, value, kernel_size, scale_factor, want_attn, halo=(0, 0)):
    """Run the fused kernel; returns (out, attn or None).  ``halo`` = extra key/value rows (top, bottom)."""
    return (_lib.host or _lib.load_host()).fused_forward_raw(query, key, value, kernel_size, scale_factor, want_attn, halo[0], halo[1])


def _nhwc_forward(query, key, value, kernel_size, scale_factor, return_attn):
    _lib.check_tensors(("value", value), ("query", query), ("key", key))
    n, hq, wq, d = query.shape
    h, w, c = value.shape[1:]
    assert key.shape == (n, h, w, d) and hq == h * scale_factor and wq == w * scale_factor
    query, key, value = _lib.aligned(query), _lib.aligned(key), _lib.aligned(value)
    out = torch.empty((n, hq, wq, c), dtype=value.dtype, device=value.device)
    attn = torch.empty((n, hq, wq, kernel_size ** 2), dtype=value.dtype, device=value.device) if return_attn else None
    _lib.call("sapa_fused_forward_nhwc", value.device, query, key, value, out, attn, n, d, c, h, w, kernel_size, scale_factor,
              _lib.dtype_code(value))
    return out, attn


class _SapaFusedNhwcFunction(Function):
    """Channels-last forward kernel; the backward goes through the channels-first kernels: the saved tensors and the
    incoming gradient are permuted to [B, C, H, W], the fused forward is run again there for its attention map, the
    fused backward follows, and the three gradients are permuted back (five layout copies and one forward more than a
    native channels-last backward would need)."""

    @staticmethod
    def forward(ctx, query, key, value, kernel_size, scale_factor):
        out, _ = _nhwc_forward(query, key, value, kernel_size, scale_factor, False)
        if any(ctx.needs_input_grad[:3]):
            ctx.cfg = (kernel_size, scale_factor)
            ctx.save_for_backward(query, key, value)
        return out

    @staticmethod
    def backward(ctx, grad_out):
        query, key, value = ctx.saved_tensors
        kernel_size, scale_factor = ctx.cfg
        first = [t.detach().permute(0, 3, 1, 2).contiguous().requires_grad_() for t in (query, key, value)]
        with torch.enable_grad():
            out = SapaFusedFunction.apply(first[0], first[1], first[2], kernel_size, scale_factor)
        grads = torch.autograd.grad(out, first, grad_out.permute(0, 3, 1, 2).contiguous())
        gq, gk, gv = (g.permute(0, 2, 3, 1).contiguous() for g in grads)
        return gq, gk, gv, None, None


def sapa_fused_nhwc(query, key, value, kernel_size=5, scale_factor=2, return_attn=False):
    """Fused SAPA-B on channels-last tensors: ``query`` [B, sH, sW, d], ``key`` [B, H, W, d], ``value`` [B, H, W, C] ->
    [B, sH, sW, C] (plus the attention [B, sH, sW, K*K] when ``return_attn``, which is not differentiable).  The forward
    is the channels-last kernel; gradients are computed by the channels-first kernels around layout copies (see
    ``_SapaFusedNhwcFunction``).  The reference has no channels-last path."""
    if not value.is_cuda:
        raise NotImplementedError
    needs_grad = torch.is_grad_enabled() and any(t.requires_grad for t in (query, key, value))
    if return_attn:
        if needs_grad:
            raise NotImplementedError("sapa_fused_nhwc(return_attn=True) is forward only")
        return _nhwc_forward(query, key, value, kernel_size, scale_factor, True)
    if needs_grad:
        return _SapaFusedNhwcFunction.apply(query, key, value, kernel_size, scale_factor)
    return _nhwc_forward(query, key, value, kernel_size, scale_factor, False)[0]
