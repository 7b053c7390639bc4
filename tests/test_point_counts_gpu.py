"""SAPA-D with any number of points: the window kernels have instances for up to 4, 8, 9 and 16 points, and half-sized blocks for small
images."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 2e-2), (torch.float16, 4e-3)])
@pytest.mark.parametrize("points", [1, 3, 4, 5, 8, 10, 15, 16])
@pytest.mark.parametrize("H,W", [(1, 8), (5, 8), (10, 16), (11, 24)])      # 32, 160, 640, 1056 pixels: half a block, a quarter over, whole blocks
def test_forward(H, W, points, dtype, tol):
    """2-norm against the float64 ops; tol as in test_outlier_lists_gpu.py."""
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, C, d, G = 3, 12, 6, 3
    g = torch.Generator().manual_seed(points)
    q, k, v, o = (torch.randn(*s, generator=g) * f for s, f in (((B, d, 2 * H, 2 * W), 0.5), ((B, d, H, W), 0.5), ((B, C, H, W), 1.0),
                                                                ((B, 2 * points * G, 2 * H, 2 * W), 0.8)))
    o = (o * 64).round() / 64 + 1 / 128      # positions are exact in float32: the same cells as in float64
    t = [x.to(dtype).to(DEV) for x in (q, k, v, o, torch.rand(B, G, points, 2 * H, 2 * W, generator=g))]

    def results(q, k, v, o, a):
        return sp.deform_sapa_fused(q, k, v, o, points, 2, G), sp.deform_qk(q, k, o, points, 2, G), sp.deform_av(a, v, o, points, 2, G)
    got = results(*t)
    assert "deform_window_kernel<weights>" in _lib.last_kernels()
    for x, y in zip(got, results(*[x.double() for x in t])):
        assert float((x.double() - y).norm()) <= tol * float(y.norm())
