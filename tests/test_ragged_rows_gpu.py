"""Rows that are not multiples of 16 bytes: the ragged form of the tensor-core kernels (no tensor maps, boxes copied by
producer warps), at the widths and channel counts where its boxes, stores and work items end."""
import pytest
import torch

from conftest import expected_fused_backward, expected_fused_forward, rel_err

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# B, d, C, H, W: odd and even widths around the 8-column tile, one column, a channel tail, several items per tile (few tiles
# and many channels), several tiles per CTA
SHAPES = [(2, 16, 24, 7, 9), (1, 5, 7, 3, 1), (1, 40, 33, 5, 15), (1, 32, 256, 9, 18), (3, 16, 40, 33, 50)]


@pytest.mark.parametrize("dtype,tol,tol_grad", [(torch.float32, 1e-5, 2e-5), (torch.bfloat16, 1e-2, 3e-2), (torch.float16, 2e-3, 4e-3)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "B%d_d%d_C%d_%dx%d" % s)
def test_ragged_rows_vs_oracle(oracle, shape, dtype, tol, tol_grad):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, d, C, H, W = shape
    g = torch.Generator().manual_seed(3)
    q, k, v, go = (torch.randn(*s, generator=g).to(dtype) for s in ((B, d, 2 * H, 2 * W), (B, d, H, W), (B, C, H, W), (B, C, 2 * H, 2 * W)))
    q, k = (0.5 * q).to(dtype), (0.5 * k).to(dtype)
    n = [t.double().numpy() for t in (q, k, v)]
    want = oracle.sapa_forward(*n, 5, 2)
    want_g = oracle.sapa_backward(go.double().numpy(), *n, 5, 2)
    t = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    fused = sp.sapa_fused(*t, 5, 2)
    name = {torch.float32: "f32", torch.bfloat16: "bf16", torch.float16: "f16"}[dtype]
    assert _lib.last_kernels() == expected_fused_forward(5, 2, W, name, B, H, C, d)
    got = torch.autograd.grad(fused, t, go.to(DEV))
    assert _lib.last_kernels() == expected_fused_backward(5, 2, W, name, B, H, C, d)
    sep = sp.av(torch.softmax(sp.qk(t[0], t[1], 5, 2), dim=1), t[2], 5, 2)
    got_sep = torch.autograd.grad(sep, t, go.to(DEV))
    # the separate ops round the logits and the attention map too: twice the forward's bound
    for out, grads, f in ((fused, got, 1), (sep, got_sep, 2)):
        assert rel_err(out.detach().double().cpu().numpy(), want) < f * tol
        for a, b in zip(grads, want_g):
            assert rel_err(a.double().cpu().numpy(), b) < f * tol_grad
    assert _lib.wait_timeout_flags(DEV) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_odd_rows_keep_float32_weights(dtype):
    """The attention weights of rows of odd length are two terms: what the output is off by is its own rounding and little more
    (weights of one 16-bit term would add 0.9 of that rounding)."""
    import sapa_b200 as sp
    g = torch.Generator().manual_seed(8)
    q, k, v = ((torch.randn(*s, generator=g) * f).to(dtype).to(DEV) for s, f in (((2, 32, 40, 82), 0.5), ((2, 32, 20, 41), 0.5), ((2, 64, 20, 41), 1.0)))
    want = sp.sapa_fused(q.double(), k.double(), v.double(), 5, 2)
    off = [float((t.double() - want).norm()) for t in (sp.sapa_fused(q, k, v, 5, 2), want.to(dtype))]
    assert off[0] <= 1.1 * off[1]
