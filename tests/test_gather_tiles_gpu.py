"""The gather kernels (value and key gradients) at the widths, heights and channel counts where their tiles end: 4 x 32 cells in 16
bits, 4 x 8 cells in float32 and for narrow 16-bit images."""
import pytest
import torch
import torch.nn.functional as F

from conftest import expected_gath, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# B, C, H, W: one tile exactly and less of it, rows and columns of a second and third, channel tails, few channels, more items than SMs
SHAPES = [(2, 16, 4, 32), (1, 40, 7, 24), (3, 33, 17, 56), (2, 7, 15, 64), (1, 64, 16, 8), (2, 20, 33, 40), (1, 3, 1, 4), (40, 24, 18, 32)]


def _want(go, attn, value):
    """Gradient of value of out[c, p] = sum_k attn[k, p] window_k(value)[c, p], in float64."""
    v = value.double().requires_grad_()
    B, C, H, W = v.shape
    win = F.unfold(v, 5, padding=2).view(B, C, 25, H, W).repeat_interleave(2, 3).repeat_interleave(2, 4)
    return torch.autograd.grad((win * attn.double()[:, None]).sum(2), v, go.double())[0].numpy()


# float32: three-term tf32 (1e-6) over 100 products.  16 bits: exact products, float32 sums, one rounding of the result (half an ulp)
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 5e-6), (torch.bfloat16, 4e-3), (torch.float16, 1e-3)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "B%d_C%d_%dx%d" % s)
def test_gather_vs_float64(shape, dtype, tol):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, C, H, W = shape
    g = torch.Generator().manual_seed(9)
    attn, go, v = (torch.randn(*s, generator=g).to(dtype) for s in ((B, 25, 2 * H, 2 * W), (B, C, 2 * H, 2 * W), (B, C, H, W)))
    t = v.to(DEV).requires_grad_()
    got = torch.autograd.grad(sp.av(attn.to(DEV), t, 5, 2), t, go.to(DEV))[0]
    assert _lib.last_kernels()[-1] == expected_gath(5, 2, W, {torch.float32: "f32", torch.bfloat16: "bf16", torch.float16: "f16"}[dtype], H, C)
    assert rel_err(got.double().cpu().numpy(), _want(go, attn, v)) < tol
    assert _lib.wait_timeout_flags(DEV) == 0
