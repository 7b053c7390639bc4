"""Points outside the 5 x 5 window of their pixel: a short list (a warp per entry, side buffers touched cell by cell), a long one, and
two points that share cells, forward and backward against the float64 ops."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 2e-2), (torch.float16, 4e-3)])
@pytest.mark.parametrize("sigma", [0.2, 0.6, 1.5])      # no other point, about a thousand, about a hundred thousand listed
@pytest.mark.parametrize("B,C,d,H,W,G", [(2, 96, 24, 48, 40, 4), (1, 5, 1, 48, 40, 1)])
def test_listed_points(B, C, d, H, W, G, sigma, dtype, tol):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    g = torch.Generator().manual_seed(4)
    q, k, v, o, go = (torch.randn(*s, generator=g) * f for s, f in (((B, d, 2 * H, 2 * W), 0.5), ((B, d, H, W), 0.5), ((B, C, H, W), 1.0),
                                                                    ((B, 18 * G, 2 * H, 2 * W), sigma), ((B, C, 2 * H, 2 * W), 1.0)))
    o = (o * 64).round() / 64 + 1 / 128      # positions are exact in float32: the same cells as in float64
    o[0, :2, 10, 10:14] = 3.25        # the same point for two pixels of two parents
    t = [x.to(dtype).to(DEV).requires_grad_() for x in (q, k, v, o)]
    r = [x.detach().double().requires_grad_() for x in t]
    out, want = sp.deform_sapa_fused(*t, 9, 2, G), sp.deform_sapa_fused(*r, 9, 2, G)
    got = torch.autograd.grad(out, t, go.to(dtype).to(DEV))
    ref = torch.autograd.grad(want, r, go.to(dtype).to(DEV).double())
    # 2-norms.  float32: a few hundred products and exponentials.  16 bits: attention, windows and gradients rounded on the way
    for a, b in zip([out, *got], [want, *ref]):
        assert float((a.detach().double() - b.detach()).norm() / b.detach().norm()) < tol
    assert _lib.wait_timeout_flags(DEV) == 0
