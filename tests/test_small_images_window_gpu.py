"""SAPA-D on images whose pixels end in the first half of a block of the window kernels: blocks of half the size, in training too."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 2e-2), (torch.float16, 4e-3)])      # as in test_outlier_lists_gpu.py
@pytest.mark.parametrize("H,W", [(1, 8), (2, 8), (3, 16), (5, 16), (7, 16), (4, 16)])      # 32, 64, 192, 320, 448 pixels; 256: whole blocks
def test_small_images(H, W, dtype, tol):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, C, d, G, P = 5, 12, 8, 4, 9
    g = torch.Generator().manual_seed(H)
    q, k, v, o, go = (torch.randn(*s, generator=g) * f for s, f in (((B, d, 2 * H, 2 * W), 0.5), ((B, d, H, W), 0.5), ((B, C, H, W), 1.0),
                                                                    ((B, 2 * P * G, 2 * H, 2 * W), 0.8), ((B, C, 2 * H, 2 * W), 1.0)))
    o = (o * 64).round() / 64 + 1 / 128      # positions are exact in float32: the same cells as in float64
    t = [x.to(dtype).to(DEV).requires_grad_() for x in (q, k, v, o)]
    r = [x.detach().double().requires_grad_() for x in t]
    out, want = sp.deform_sapa_fused(*t, P, 2, G), sp.deform_sapa_fused(*r, P, 2, G)
    up = go.to(dtype).to(DEV)
    for n, (x, y) in enumerate(zip((out, *torch.autograd.grad(out, t, up)), (want, *torch.autograd.grad(want, r, up.double())))):
        assert float((x.double() - y).norm()) <= tol * float(y.norm()), n
    assert _lib.wait_timeout_flags(DEV) == 0
