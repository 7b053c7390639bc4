"""The 4 x 32 tiles of the 16-bit tensor-core kernel (batches of images at least 24 pixels wide): all four modes, at the widths,
heights and channel counts where its tiles, boxes and stages end."""
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# B, d, C, H, W: at least 128 tiles each; one tile 24 columns wide, a second tile of 24 columns, rows and channel tails, two items
# per CTA and more
SHAPES = [(32, 16, 40, 14, 24), (16, 24, 72, 15, 56), (8, 40, 33, 64, 64)]


@pytest.mark.parametrize("dtype,tol,tol_grad", [(torch.bfloat16, 1e-2, 3e-2), (torch.float16, 2e-3, 4e-3)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "B%d_d%d_C%d_%dx%d" % s)
def test_wide_tiles_vs_oracle(oracle, shape, dtype, tol, tol_grad):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, d, C, H, W = shape
    g = torch.Generator().manual_seed(5)
    q, k, v, go = (torch.randn(*s, generator=g).to(dtype) for s in ((B, d, 2 * H, 2 * W), (B, d, H, W), (B, C, H, W), (B, C, 2 * H, 2 * W)))
    q, k = (0.5 * q).to(dtype), (0.5 * k).to(dtype)
    n = [t.float().numpy() for t in (q, k, v)]
    want = oracle.sapa_forward(*n, 5, 2)
    want_g = oracle.sapa_backward(go.float().numpy(), *n, 5, 2)
    t = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    fused = sp.sapa_fused(*t, 5, 2)
    got = torch.autograd.grad(fused, t, go.to(DEV))
    with torch.no_grad():       # a single image has too few tiles: the 4 x 8 tiles, same bits
        one = sp.sapa_fused(q[3:4].to(DEV), k[3:4].to(DEV), v[3:4].to(DEV), 5, 2)
    assert torch.equal(one[0], fused[3])
    sep = sp.av(torch.softmax(sp.qk(t[0], t[1], 5, 2), dim=1), t[2], 5, 2)
    got_sep = torch.autograd.grad(sep, t, go.to(DEV))
    # the separate ops round the logits and the attention map too: twice the forward's bound
    for out, grads, f in ((fused, got, 1), (sep, got_sep, 2)):
        assert rel_err(out.detach().float().cpu().numpy(), want) < f * tol
        for a, b in zip(grads, want_g):
            assert rel_err(a.float().cpu().numpy(), b) < f * tol_grad
    assert _lib.wait_timeout_flags(DEV) == 0
