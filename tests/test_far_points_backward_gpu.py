"""The per-pixel step of SAPA-D's backward with few and many points outside the window in a warp (gathered by the warp together and by each
thread), every count of points of its instances, pixels that end inside a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 2e-2), (torch.float16, 4e-3)])      # as in test_outlier_lists_gpu.py
@pytest.mark.parametrize("points,far", [(1, 0.02), (4, 0.004), (5, 0.05), (8, 0.3), (9, 0.004), (9, 0.06), (9, 1.0), (16, 0.01), (16, 0.5)])
def test_far_points(points, far, dtype, tol):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, C, d, H, W, G = 2, 70, 14, 9, 24, 2
    g = torch.Generator().manual_seed(points)
    q, k, v, o, go = (torch.randn(*s, generator=g) * f for s, f in (((B, d, 2 * H, 2 * W), 0.5), ((B, d, H, W), 0.5), ((B, C, H, W), 1.0),
                                                                    ((B, 2 * points * G, 2 * H, 2 * W), 0.4), ((B, C, 2 * H, 2 * W), 1.0)))
    moved = torch.rand(o.shape, generator=g) < far
    o = torch.where(moved, 3.0 * torch.sign(o), o.clamp(-1.5, 1.5))
    o = (o * 64).round() / 64 + 1 / 128      # positions are exact in float32: the same cells as in float64
    t = [x.to(dtype).to(DEV).requires_grad_() for x in (q, k, v, o)]
    r = [x.detach().double().requires_grad_() for x in t]
    a = torch.softmax(torch.randn(B, G, points, 2 * H, 2 * W, generator=g), 2).to(dtype).to(DEV).requires_grad_()
    ra, up = a.detach().double().requires_grad_(), go.to(dtype).to(DEV)
    got = torch.autograd.grad(sp.deform_sapa_fused(*t, points, 2, G), t, up) + torch.autograd.grad(sp.deform_av(a, t[2], t[3], points, 2, G), (a, t[2], t[3]), up)
    want = torch.autograd.grad(sp.deform_sapa_fused(*r, points, 2, G), r, up.double()) \
        + torch.autograd.grad(sp.deform_av(ra, r[2], r[3], points, 2, G), (ra, r[2], r[3]), up.double())
    for n, (x, y) in enumerate(zip(got, want)):
        assert float((x.double() - y).norm()) <= tol * (float(y.norm()) or 1.0), n
    assert _lib.wait_timeout_flags(DEV) == 0
