"""Operators of SAPA-D: ``deform_qk``, ``deform_av`` and the fused ``deform_sapa_fused``.

Names, positional arguments and assertions follow ``DeformQKFunction`` / ``DeformAVFunction`` of the
reference (deformsapa/deformsapa/deform_func.py:7-114).  Checks, allocation, the choice between the dense-window and the
gather kernels and the autograd nodes are native (``csrc/host.cpp``, ``csrc/host_deform.inc``); the ``Function`` classes run the
same native code for traces and transforms (``_lib.transformed``), and for callers who use them by name.
"""
from __future__ import annotations

import torch
from torch.autograd import Function

from . import _lib


def deform_qk(query, key, offset, num_point, scale_factor, groups):
    """out[b,g,p,qh,qw] = <query_g[b,:,qh,qw], bilinear(key_g[b], (qh/s, qw/s) + offset[b,g,p])>."""
    if _lib.transformed():
        return DeformQKFunction.apply(query, key, offset, num_point, scale_factor, groups)
    return (_lib.host or _lib.load_host()).deform_qk(query, key, offset, num_point, scale_factor, groups)


def deform_av(attn, value, offset, num_point, scale_factor, groups):
    """out[b,c,qh,qw] = sum_p attn[b,g(c),p,qh,qw] * bilinear(value[b,c], (qh/s, qw/s) + offset[b,g(c),p])."""
    if _lib.transformed():
        return DeformAVFunction.apply(attn, value, offset, num_point, scale_factor, groups)
    return (_lib.host or _lib.load_host()).deform_av(attn, value, offset, num_point, scale_factor, groups)


def deform_sapa_fused(query, key, value, offset, num_point=9, scale_factor=2, groups=4):
    """deform_av(softmax_p(deform_qk(q, k, offset)), v, offset) as one op (``SAPADeform.attention``, sapa_deform.py:51-53);
    differentiable with respect to query, key, value and offset."""
    if _lib.transformed():
        return DeformSapaFusedFunction.apply(query, key, value, offset, num_point, scale_factor, groups)
    return (_lib.host or _lib.load_host()).deform_sapa_fused(query, key, value, offset, num_point, scale_factor, groups)


class DeformQKFunction(Function):
    """``deform_qk`` under the name that the reference exposes."""

    @staticmethod
    def forward(ctx, query, key, offset, num_point, scale_factor, groups):
        ctx.points = (num_point, scale_factor, groups)
        ctx.save_for_backward(query, key, offset)
        return _lib.load_host().deform_qk(query, key, offset, num_point, scale_factor, groups)

    @staticmethod
    def backward(ctx, grad_output):
        return (*_lib.load_host().deform_qk_backward(grad_output, *ctx.saved_tensors, *ctx.points), None, None, None)


class DeformAVFunction(Function):
    """``deform_av`` under the name that the reference exposes."""

    @staticmethod
    def forward(ctx, attn, value, offset, num_point, scale_factor, groups):
        ctx.points = (num_point, scale_factor, groups)
        ctx.save_for_backward(attn, value, offset)
        return _lib.load_host().deform_av(attn, value, offset, num_point, scale_factor, groups)

    @staticmethod
    def backward(ctx, grad_output):
        return (*_lib.load_host().deform_av_backward(grad_output, *ctx.saved_tensors, *ctx.points), None, None, None)


class DeformSapaFusedFunction(Function):
    @staticmethod
    def forward(ctx, query, key, value, offset, num_point, scale_factor, groups):
        ctx.points = (num_point, scale_factor, groups)
        out, attn = _lib.load_host().deform_fused_forward(query, key, value, offset, num_point, scale_factor, groups, any(ctx.needs_input_grad[:4]))
        if attn is not None:
            ctx.save_for_backward(query, key, value, offset, attn)
        return out

    @staticmethod
    def backward(ctx, grad_output):
        return (*_lib.load_host().deform_fused_backward(grad_output, *ctx.saved_tensors, *ctx.points), None, None, None)


def deform_fused_supported(num_point: int, dtype: torch.dtype) -> bool:
    return num_point <= 16 and dtype in (torch.float32, torch.float16, torch.bfloat16)


def _dense_workspace_bytes(t, n, h, w, num_point, scale_factor, groups, others=()) -> int:
    """Workspace of the dense-window forward kernels for this problem, 0 when they do not apply (they need s = 2 and
    float32, or float16 / bfloat16 with rows of 16 bytes and every tensor of the call - ``t`` and ``others`` - on a
    16-byte boundary)."""
    if t.dtype not in (torch.float32, torch.float16, torch.bfloat16) or num_point > 16 or t.data_ptr() % 16 != 0:
        return 0
    if t.dtype != torch.float32 and any(o.data_ptr() % 16 != 0 for o in others):
        return 0
    return int(_lib.lib().sapa_deform_fused_forward_workspace(n, h, w, num_point, scale_factor, groups, _lib.dtype_code(t)))
