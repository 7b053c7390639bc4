"""The 4 x 32 tiles of the 16-bit tensor-core kernel (batches of images at least 24 pixels wide): all four modes, at the widths,
heights and channel counts where its tiles, boxes and stages end."""
import pytest
import torch

from conftest import expected_agg, expected_fused_backward, expected_fused_forward, expected_gath, expected_sim, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# B, d, C, H, W: at least 100 tiles each, from where the wide ones are taken; one tile 24 columns wide, a second tile of 24 columns, rows and channel tails, two items
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
    assert _lib.last_kernels() == ["sapa_wide_16_kernel<fwd>"]
    got = torch.autograd.grad(fused, t, go.to(DEV))
    assert _lib.last_kernels() == ["sapa_wide_16_kernel<bwd>"] + ["sapa_gath_wide_16_kernel"] * 2
    with torch.no_grad():       # a single image has too few tiles: the 4 x 8 tiles, same bits
        one = sp.sapa_fused(q[3:4].to(DEV), k[3:4].to(DEV), v[3:4].to(DEV), 5, 2)
        assert _lib.last_kernels() == ["sapa_tma_fused_16_kernel<fwd>"]
    assert torch.equal(one[0], fused[3])
    sep = sp.av(torch.softmax(sp.qk(t[0], t[1], 5, 2), dim=1), t[2], 5, 2)
    got_sep = torch.autograd.grad(sep, t, go.to(DEV))
    # the separate ops round the logits and the attention map too: twice the forward's bound
    for out, grads, f in ((fused, got, 1), (sep, got_sep, 2)):
        assert rel_err(out.detach().float().cpu().numpy(), want) < f * tol
        for a, b in zip(grads, want_g):
            assert rel_err(a.float().cpu().numpy(), b) < f * tol_grad
    assert _lib.wait_timeout_flags(DEV) == 0


# images and sizes on either side of the rules: 99 and 100 tiles, three quarters of one and of two tiles' columns and eight columns
# less, rows of 16 bytes and others
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,H,W", [(99, 4, 32), (100, 4, 32), (33, 9, 24), (34, 9, 24), (100, 4, 16), (50, 4, 48), (60, 4, 40), (2, 3, 36), (2, 3, 34), (2, 3, 33)])
def test_which_kernel_serves(B, H, W, dtype):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    name = {torch.bfloat16: "bf16", torch.float32: "f32"}[dtype]
    q, k, v, a = (torch.randn(*s, device=DEV).to(dtype).requires_grad_() for s in ((B, 8, 2 * H, 2 * W), (B, 8, H, W), (B, 8, H, W), (B, 25, 2 * H, 2 * W)))
    out = sp.sapa_fused(q, k, v, 5, 2)
    assert _lib.last_kernels() == expected_fused_forward(5, 2, W, name, B, H)
    torch.autograd.grad(out.sum(), (q, k, v))
    assert _lib.last_kernels() == expected_fused_backward(5, 2, W, name, B, H)
    sim, agg = expected_sim(5, 2, W, name, B, H), expected_agg(5, 2, W, name, B, H)
    out = sp.qk(q, k, 5, 2)
    assert _lib.last_kernels() == sim
    torch.autograd.grad(out.sum(), (q, k))
    assert _lib.last_kernels() == agg + [expected_gath(5, 2, W, name)]
    out = sp.av(a, v, 5, 2)
    assert _lib.last_kernels() == agg
    torch.autograd.grad(out.sum(), (a, v))
    assert _lib.last_kernels() == sim + [expected_gath(5, 2, W, name)]
