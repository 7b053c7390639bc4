"""GroupNorm + 1x1 projection in front of the attention (``self.q(self.norm_y(y))`` / ``self.k(self.norm_x(x))`` of the
reference modules, sapa_base.py:27-34, sapa_deform.py:35-42) as one tensor-core GEMM: ``sapa_project_forward`` of the C ABI.

Forward only; the modules reach this kernel, and the ones that are differentiable, through their native path.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from . import _lib


def project_supported(x: torch.Tensor, norm, conv: nn.Conv2d) -> bool:
    """True when :func:`project` can run this projection (CUDA, float32 / float16 / bfloat16, 1x1 convolution with
    stride 1 and one group, a shape the GEMM kernel takes)."""
    if not x.is_cuda or x.dim() != 4 or x.dtype not in (torch.float32, torch.float16, torch.bfloat16):
        return False
    if conv.kernel_size != (1, 1) or conv.stride != (1, 1) or conv.padding != (0, 0) or conv.groups != 1 or conv.dilation != (1, 1):
        return False
    if norm is not None and not isinstance(norm, nn.GroupNorm):
        return False
    if norm is not None and not norm.affine:
        return False
    return _lib.load_host().project_workspace(x, norm.num_groups if norm is not None else 0, conv.weight) != 0


def project(x: torch.Tensor, norm, conv: nn.Conv2d) -> torch.Tensor:
    """``conv(norm(x))`` for a 1x1 ``conv`` and a GroupNorm (or ``None``) ``norm``; ``x`` [B, C, H, W] -> [B, d, H, W]."""
    if norm is None:
        return _lib.load_host().project(x, None, None, 0, 0.0, conv.weight, conv.bias)
    return _lib.load_host().project(x, norm.weight, norm.bias, norm.num_groups, norm.eps, conv.weight, conv.bias)
