"""The 16-bit similarity on strips of columns, by itself and with the softmax backward behind it (stage 1 of the fused backward): channels
that fill a stage partly, odd rows, partial strips, several units a CTA."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(seed, *shape, dtype, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype).to(DEV)


def _windows(t):
    H, W = t.shape[2:]
    padded = F.pad(t, (2, 2, 2, 2))
    return [padded[:, :, i // 5:i // 5 + H, i % 5:i % 5 + W].repeat_interleave(2, 2).repeat_interleave(2, 3) for i in range(25)]


def _off(a, b):
    return float((a.double() - b).norm() / b.norm())


# one rounding of a float32 sum: half an ulp at most, 0.3 of one in the mean (1.7e-3, 2.1e-4)
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2e-3), (torch.float16, 2.5e-4)])
@pytest.mark.parametrize("shape", [(1, 1, 1, 8), (2, 16, 7, 40), (3, 17, 33, 72), (70, 32, 5, 24), (1, 100, 150, 264)], ids=lambda s: "B%d_d%d_%dx%d" % s)
def test_similarity(shape, dtype, tol):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, d, H, W = shape
    q, k = _rand(1, B, d, 2 * H, 2 * W, dtype=dtype, scale=0.5), _rand(2, B, d, H, W, dtype=dtype, scale=0.5)
    want = torch.stack([(q.double() * w).sum(1) for w in _windows(k.double())], 1)
    for _ in range(2):
        got = sp.qk(q, k, 5, 2)
        assert _lib.last_kernels() == ["sapa_strip_sim_16_kernel<logits>"]
        assert _off(got, want) < tol and float((got.double() - want).abs().max() / want.abs().max()) < 4 * tol
    assert _lib.wait_timeout_flags(DEV) == 0


# the attention map, the logit gradients and the result are rounded: 2.8e-3 and 3.6e-4 measured, as on the tiles
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 4e-3), (torch.float16, 5e-4)])
@pytest.mark.parametrize("shape", [(1, 128, 20, 9, 16), (2, 150, 32, 33, 40), (5, 300, 64, 21, 72), (48, 48, 7, 30, 32)], ids=lambda s: "B%d_C%d_d%d_%dx%d" % s)
def test_backward(shape, dtype, tol):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, C, d, H, W = shape
    t = [_rand(1, B, d, 2 * H, 2 * W, dtype=dtype, scale=0.5), _rand(2, B, d, H, W, dtype=dtype, scale=0.5), _rand(3, B, C, H, W, dtype=dtype)]
    go = _rand(4, B, C, 2 * H, 2 * W, dtype=dtype)
    r = [x.double().requires_grad_() for x in t]
    attn = torch.softmax(torch.stack([(r[0] * w).sum(1) for w in _windows(r[1])], 1), 1)
    grads = torch.autograd.grad(sum(attn[:, i:i + 1] * w for i, w in enumerate(_windows(r[2]))), r, go.double())
    t = [x.requires_grad_() for x in t]
    for _ in range(2):
        for a, b in zip(torch.autograd.grad(sp.sapa_fused(*t, 5, 2), t, go), grads):
            assert _off(a, b) < tol
        # rows of 16 columns are left to the tiles
        assert _lib.last_kernels()[:2] == ["sapa_strip_sim_16_kernel<softmax_bwd>", "sapa_strip_kernel"] or W == 16
    assert _lib.wait_timeout_flags(DEV) == 0
