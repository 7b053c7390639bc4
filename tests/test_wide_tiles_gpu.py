"""The 4 x 32 tiles of the 16-bit tensor-core kernel (batches of images at least 24 pixels wide): all four modes, at the widths,
heights and channel counts where its tiles, boxes and stages end."""
import pytest
import torch

from conftest import expected_agg, expected_fused_backward, expected_fused_forward, expected_gath, expected_sim, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# B, d, C, H, W: at least 100 tiles each, from where the wide ones are taken; one tile 24 columns wide, a second tile of 24 columns, rows and channel tails, two items
# per CTA and more.  The last four stay off the strips: forward with more than 64 query channels, with few value channels, all modes but the similarity
SHAPES = [(32, 16, 40, 14, 24), (16, 24, 72, 15, 56), (8, 40, 33, 64, 64), (16, 80, 24, 15, 56), (8, 72, 30, 64, 64), (8, 96, 72, 40, 56), (32, 8, 12, 14, 24)]


@pytest.mark.parametrize("dtype,tol,tol_grad", [(torch.bfloat16, 1e-2, 3e-2), (torch.float16, 2e-3, 4e-3)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "B%d_d%d_C%d_%dx%d" % s)
def test_wide_tiles_vs_oracle(oracle, shape, dtype, tol, tol_grad):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    from sapa_b200.functions import fused_forward_raw
    B, d, C, H, W = shape
    g = torch.Generator().manual_seed(5)
    q, k, v, go = (torch.randn(*s, generator=g).to(dtype) for s in ((B, d, 2 * H, 2 * W), (B, d, H, W), (B, C, H, W), (B, C, 2 * H, 2 * W)))
    q, k = (0.5 * q).to(dtype), (0.5 * k).to(dtype)
    n = [t.float().numpy() for t in (q, k, v)]
    name = {torch.bfloat16: "bf16", torch.float16: "f16"}[dtype]
    want, want_attn = oracle.sapa_forward(*n, 5, 2, return_attn=True)
    want_g = oracle.sapa_backward(go.float().numpy(), *n, 5, 2)
    t = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    fused = sp.sapa_fused(*t, 5, 2)
    forward = _lib.last_kernels()
    assert forward == expected_fused_forward(5, 2, W, name, B, H, C, d) == (["sapa_wide_16_kernel<fwd>"] if d > 64 or C * H * W < 2e4 else ["sapa_strip_fwd_kernel"])
    got = torch.autograd.grad(fused, t, go.to(DEV))
    assert _lib.last_kernels() == expected_fused_backward(5, 2, W, name, B, H, C, d)
    if C < 32:
        assert _lib.last_kernels()[0] == "sapa_wide_16_kernel<bwd>" and _lib.last_kernels()[-1] == "sapa_gath_wide_16_kernel"
    with torch.no_grad():       # a single image has too few tiles: the 4 x 8 tiles, same bits
        one = sp.sapa_fused(q[3:4].to(DEV), k[3:4].to(DEV), v[3:4].to(DEV), 5, 2)
        assert _lib.last_kernels() == (["sapa_tma_fused_16_kernel<fwd>"] if "wide" in forward[0] else forward)
    assert torch.equal(one[0], fused[3])
    out, attn = fused_forward_raw(*(x.detach() for x in t), 5, 2, True)
    assert torch.equal(out, fused) and rel_err(attn.float().cpu().numpy(), want_attn) < tol
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
    assert _lib.last_kernels() == agg + [expected_gath(5, 2, W, name, H)]
    out = sp.av(a, v, 5, 2)
    assert _lib.last_kernels() == agg
    torch.autograd.grad(out.sum(), (a, v))
    assert _lib.last_kernels() == sim + [expected_gath(5, 2, W, name, H)]


# either side of the lines between tiles and strips (channels of value and query, rows, columns): values of an image, columns inside the strips, channels; tall
# and flat images, batches that must not matter
LINES = [(1, 24, 16, 27, 32), (1, 24, 16, 26, 32), (1, 24, 64, 40, 32), (1, 24, 65, 40, 32), (1, 23, 16, 64, 32), (4, 100, 16, 20, 16), (4, 100, 16, 20, 8),
         (1, 48, 16, 128, 128), (1, 48, 16, 40, 160), (1, 96, 16, 73, 72), (1, 96, 16, 73, 76), (1, 47, 16, 128, 128), (1, 256, 16, 4, 64), (8, 256, 16, 4, 64),
         (1, 64, 64, 30, 32), (1, 64, 64, 29, 32), (16, 64, 64, 29, 32), (1, 63, 32, 64, 64), (2, 64, 64, 40, 20), (2, 64, 64, 40, 24), (1, 32, 32, 30, 32),
         (1, 32, 32, 29, 32), (1, 32, 32, 64, 40), (1, 31, 16, 64, 40), (2, 16, 16, 40, 16), (2, 256, 64, 15, 16), (2, 256, 64, 14, 16), (1, 16, 16, 25, 24),
         (1, 16, 16, 27, 24), (1, 16, 16, 40, 16), (1, 104, 64, 24, 40), (1, 105, 64, 24, 40), (1, 72, 8, 2800, 512), (1, 64, 8, 2800, 512)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,C,d,H,W", LINES)
def test_tiles_or_strips(B, C, d, H, W, dtype):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    name = {torch.bfloat16: "bf16", torch.float32: "f32"}[dtype]
    q, k, v, a = (torch.randn(*s, device=DEV, dtype=dtype).requires_grad_() for s in ((B, d, 2 * H, 2 * W), (B, d, H, W), (B, C, H, W), (B, 25, 2 * H, 2 * W)))
    with torch.no_grad():
        sp.sapa_fused(q, k, v, 5, 2)
        want, ran = expected_fused_forward(5, 2, W, name, B, H, C, d), _lib.last_kernels()
        assert ran == want * (len(ran) // len(want))      # once for each part that the scratch of float32 holds
    if H > 1000:
        return
    out = sp.sapa_fused(q, k, v, 5, 2)
    assert _lib.last_kernels() == expected_fused_forward(5, 2, W, name, B, H, C, d)
    torch.autograd.grad(out.sum(), (q, k, v))
    assert _lib.last_kernels() == expected_fused_backward(5, 2, W, name, B, H, C, d)
    out = sp.qk(q, k, 5, 2)
    assert _lib.last_kernels() == expected_sim(5, 2, W, name, B, H, d)
    torch.autograd.grad(out.sum(), (q, k))
    assert _lib.last_kernels() == expected_agg(5, 2, W, name, B, H, d) + [expected_gath(5, 2, W, name, H, d)]
    out = sp.av(a, v, 5, 2)
    assert _lib.last_kernels() == expected_agg(5, 2, W, name, B, H, C)
    torch.autograd.grad(out.sum(), (a, v))
    assert _lib.last_kernels() == expected_sim(5, 2, W, name, B, H, C) + [expected_gath(5, 2, W, name, H, C)]
