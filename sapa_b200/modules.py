"""``SAPA`` and ``SAPADeform``: the upsampling modules of the reference with the same constructor arguments
and parameter names, so that reference checkpoints load unchanged (``norm_y.*``, ``norm_x.*``, ``q.*``,
``k.*`` and ``offset.*``; sapa_base.py:7-49, sapa_deform.py:7-62).

One extra keyword, ``impl``: ``"fused"`` (default) runs the attention as one kernel, ``"separate"`` keeps the
reference's three steps ``qk -> F.softmax -> av`` on this library's kernels.
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.nn.modules.module import _has_any_global_hook
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext

from . import _lib
from .deform_functions import deform_av, deform_qk, deform_sapa_fused
from .functions import av, qk, sapa_fused


def _init_projection(module: nn.Module) -> None:
    # 1x1 projections start as N(0, 0.02^2) with zero bias (sapa_base.py:42-46)
    if isinstance(module, nn.Conv2d):
        nn.init.normal_(module.weight, std=0.02)
        if module.bias is not None:
            nn.init.constant_(module.bias, 0)


def _check_impl(impl: str) -> str:
    if impl not in ("fused", "separate"):
        raise ValueError(f"impl must be 'fused' or 'separate', got {impl!r}")
    return impl


def _common_dtype(*tensors):
    """Under ``torch.autocast`` the 1x1 projections come out in the autocast type while the value (the module's
    un-normalised input) keeps the caller's type; the kernels want one element type, so everything is cast to the
    autocast type.  Outside autocast the tensors pass through untouched (mismatches are then reported by the op).
    The reference modules have no autocast handling (sapa_base.py:26-40, sapa_deform.py:34-53)."""
    if tensors[0].is_cuda and torch.is_autocast_enabled():
        dtype = torch.get_autocast_dtype("cuda")
        return tuple(t.to(dtype) for t in tensors)
    return tensors


_PLAIN = (torch.Tensor, nn.Parameter, type(None))
_NO_NORM = (None, None, 0, 0.0)


def _plain(module, cls):
    """A ``cls`` with nothing around it that only calling it would run: no hooks, no ``forward`` of its own."""
    return type(module) is cls and not (module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or
                                        module._backward_pre_hooks or "forward" in module.__dict__)


def _norm_args(norm):
    """(gamma, beta, groups, eps) of a GroupNorm (or of none) for the native module path, None when it is something else."""
    if norm is None:
        return _NO_NORM
    if not _plain(norm, nn.GroupNorm) or norm.weight is None:
        return None
    return norm.weight, norm.bias, norm.num_groups, norm.eps


def _is_projection(conv):
    return (_plain(conv, nn.Conv2d) and conv.kernel_size == (1, 1) and conv.stride == (1, 1) and conv.padding == (0, 0) and
            conv.groups == 1)


def _native(*tensors):
    """Whether the native module path may run at all for these inputs and parameters (or None): not for the CPU, nor where only
    torch's own ops are seen - traces, transforms, hooks on every module, torch-function and torch-dispatch modes (a default
    device aside) - nor for subclasses of Tensor, whose elements may lie anywhere."""
    return (tensors[0].is_cuda and not _lib.transformed() and not _has_any_global_hook() and
            torch._C._len_torch_dispatch_stack() == 0 and
            (torch._C._len_torch_function_stack() == 0 or all(type(m) is DeviceContext for m in _get_current_function_mode_stack())) and
            all(type(t) in _PLAIN for t in tensors))


def _autocast_dtype():
    return torch.get_autocast_dtype("cuda") if torch.is_autocast_enabled() else None


def _projected(x, norm, conv, fuse):
    """``conv(norm(x))``: with ``fuse`` GroupNorm and the 1x1 convolution run on this library's GEMM kernels, forward and
    backward; otherwise, and for what those do not take, on the torch modules."""
    if fuse and x.is_cuda:
        args = _norm_args(norm)
        if args is not None and _is_projection(conv) and _native(x, *args[:2], conv.weight, conv.bias):
            out = (_lib.host or _lib.load_host()).project_module(x, *args, conv.weight, conv.bias, _autocast_dtype())
            if out is not None:
                return out
    return conv(norm(x)) if norm is not None else conv(x)


def _native_module(module, y, x, convs, *args):
    """The whole module in one call (``csrc/host_module.inc``): its projections and the attention.  None where that does not
    apply: another type or shape than the kernels take, replaced or hooked submodules, another ``attention`` than the class's,
    parameters of another type than the input in training."""
    if not x.is_cuda or getattr(module.attention, "__func__", None) not in _ATTENTIONS:
        return None
    norms = (_norm_args(module.norm_y), _norm_args(module.norm_x)) if module.norm else (_NO_NORM, _NO_NORM)
    if None in norms or not all(_is_projection(c) for c in convs):
        return None
    params = [p for c in convs for p in (c.weight, c.bias)]
    if not _native(x, y, *norms[0][:2], *norms[1][:2], *params):
        return None
    host = _lib.host or _lib.load_host()
    call = host.sapa_module if len(convs) == 2 else host.deform_module
    return call(y, x, *norms[0], *norms[1], *params, *args, _autocast_dtype())


class SAPA(nn.Module):
    """Similarity-aware point affiliation upsampler (SAPA-B): x (low-res) is upsampled under guidance of y."""

    def __init__(self, dim_y, dim_x=None, up_factor=2, up_kernel_size=5, embedding_dim=32, qkv_bias=True, norm=True,
                 impl="fused"):
        super().__init__()
        dim_x = dim_y if dim_x is None else dim_x
        self.up_factor, self.up_kernel_size, self.embedding_dim = up_factor, up_kernel_size, embedding_dim
        self.norm, self.impl = norm, _check_impl(impl)
        self.fuse_projection = impl == "fused"      # set to False to keep torch's GroupNorm + convolution
        if norm:
            self.norm_y = nn.GroupNorm(32, dim_y)
            self.norm_x = nn.GroupNorm(32, dim_x)
        self.q = nn.Conv2d(dim_y, embedding_dim, kernel_size=1, bias=qkv_bias)
        self.k = nn.Conv2d(dim_x, embedding_dim, kernel_size=1, bias=qkv_bias)
        self.apply(_init_projection)

    def forward(self, y, x):
        # the value is the un-normalised x; only the key is computed from the normalised one
        if self.fuse_projection and self.impl == "fused":
            out = _native_module(self, y, x, (self.q, self.k), self.up_kernel_size, self.up_factor)
            if out is not None:
                return out
        q = _projected(y, self.norm_y if self.norm else None, self.q, self.fuse_projection)
        k = _projected(x, self.norm_x if self.norm else None, self.k, self.fuse_projection)
        return self.attention(q, k, x)

    def attention(self, q, k, v):
        q, k, v = _common_dtype(q, k, v)
        if self.impl == "fused":
            return sapa_fused(q.contiguous(), k.contiguous(), v.contiguous(), self.up_kernel_size, self.up_factor)
        attn = F.softmax(qk(q, k, self.up_kernel_size, self.up_factor), dim=1)
        return av(attn, v, self.up_kernel_size, self.up_factor)


class SAPADeform(nn.Module):
    """Deformable variant (SAPA-D): num_point learned sampling points per group instead of a fixed window."""

    def __init__(self, dim_y, dim_x=None, up_factor=2, num_point=9, groups=4, embedding_dim=32, qkv_bias=True,
                 high_offset=True, norm=False, impl="fused"):
        super().__init__()
        dim_x = dim_y if dim_x is None else dim_x
        self.up_factor, self.num_point, self.groups = up_factor, num_point, groups
        self.embedding_dim, self.high_offset = embedding_dim, high_offset
        self.norm, self.impl = norm, _check_impl(impl)
        self.fuse_projection = impl == "fused"
        if norm:
            self.norm_y = nn.GroupNorm(32, dim_y)
            self.norm_x = nn.GroupNorm(32, dim_x)
        self.q = nn.Conv2d(dim_y, groups * embedding_dim, kernel_size=1, bias=qkv_bias)
        self.k = nn.Conv2d(dim_x, groups * embedding_dim, kernel_size=1, bias=qkv_bias)
        offset_dim = groups * num_point * 2 * (up_factor ** 2 if high_offset else 1)
        self.offset = nn.Conv2d(dim_x, offset_dim, kernel_size=1, bias=qkv_bias)
        self.apply(_init_projection)

    def forward(self, y, x):
        if self.fuse_projection and self.impl == "fused":
            out = _native_module(self, y, x, (self.q, self.k, self.offset), self.high_offset, self.num_point, self.up_factor, self.groups)
            if out is not None:
                return out
        q = _projected(y, self.norm_y if self.norm else None, self.q, self.fuse_projection)
        k = _projected(x, self.norm_x if self.norm else None, self.k, self.fuse_projection)
        raw = self.offset(self.norm_x(x) if self.norm else x)
        if self.high_offset:   # one offset per high-res pixel, unpacked from channels
            offset = F.pixel_shuffle(raw, upscale_factor=self.up_factor)
        else:                  # every high-res pixel of a parent shares the parent's offset
            offset = F.interpolate(raw, scale_factor=self.up_factor)
        return self.attention(q, k, x, offset)

    def attention(self, q, k, x, offset):
        q, k, x, offset = _common_dtype(q, k, x, offset)
        if self.impl == "fused":
            return deform_sapa_fused(q.contiguous(), k.contiguous(), x.contiguous(), offset.contiguous(),
                                     self.num_point, self.up_factor, self.groups)
        attn = F.softmax(deform_qk(q, k, offset, self.num_point, self.up_factor, self.groups), dim=2)
        return deform_av(attn, x, offset, self.num_point, self.up_factor, self.groups)


_ATTENTIONS = (SAPA.attention, SAPADeform.attention)      # what the native module path stands for
