"""float32 on strips of columns: logits on the 5th-generation tensor cores with the softmax, its backward or nothing behind them, then the
aggregation - the similarity, the fused forward with and without its map, and its backward, against float64."""
import pytest
import torch
from conftest import expected_fused_backward
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# images, value channels, query channels, rows, columns: stages of channels that end early, odd rows, partial strips, many units a CTA.  Two
# million values and more, half a million an image (of square images)
SHAPES = [(4, 300, 64, 47, 44), (3, 48, 5, 51, 128), (3, 130, 33, 71, 76), (4, 720, 16, 33, 28), (4, 520, 100, 130, 32)]


def _rand(seed, *shape, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(DEV)


def _windows(t):
    H, W = t.shape[2:]
    padded = F.pad(t, (2, 2, 2, 2))
    return [padded[:, :, i // 5:i // 5 + H, i % 5:i % 5 + W].repeat_interleave(2, 2).repeat_interleave(2, 3) for i in range(25)]


# 2-norms: three-term tf32 products and the roundings toward zero of their sums; measured here (before, on tiles): logits of 64 channels 6.6e-7
# (9.2e-7), output 1.1e-6 (1.5e-6), gradients up to 3.0e-6 (3.5e-6); a channel adds up to 1e-8
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "B%d_C%d_d%d_%dx%d" % s)
def test_strips_vs_float64(shape):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    from sapa_b200.functions import fused_forward_raw
    B, C, d, H, W = shape
    assert _lib.lib().sapa_fused_forward_wants_map(B, d, C, H, W, 5, 2, 0) == 1
    t = [_rand(1, B, d, 2 * H, 2 * W, scale=0.5).requires_grad_(), _rand(2, B, d, H, W, scale=0.5).requires_grad_(), _rand(3, B, C, H, W).requires_grad_()]
    go = _rand(4, B, C, 2 * H, 2 * W)
    r = [x.detach().double().requires_grad_() for x in t]
    logits = torch.stack([(r[0] * w).sum(1) for w in _windows(r[1])], 1)
    attn = torch.softmax(logits, 1)
    want = sum(attn[:, i:i + 1] * w for i, w in enumerate(_windows(r[2])))
    grads = torch.autograd.grad(want, r, go.double())

    def off(a, b):
        return float((a.detach().double() - b.detach()).norm() / b.detach().norm())
    for _ in range(2):
        out = sp.sapa_fused(*t, 5, 2)
        assert _lib.last_kernels() == ["sapa_strip_sim_kernel<softmax>", "sapa_strip_kernel"]
        got = torch.autograd.grad(out, t, go)
        assert _lib.last_kernels() == expected_fused_backward(5, 2, W, "f32", B, H, C, d)
        assert off(sp.qk(t[0].detach(), t[1].detach(), 5, 2), logits) < 5e-7 + 1e-8 * d
        assert _lib.last_kernels() == ["sapa_strip_sim_kernel<logits>"]
        assert off(out, want) < 1.3e-6 + 1e-8 * d
        for a, b in zip(got, grads):
            assert off(a, b) < 2e-6 + 1e-8 * max(C, d)
    alone, none = fused_forward_raw(*(x.detach() for x in t), 5, 2, False)
    assert none is None and torch.equal(alone, out.detach())         # with the map as scratch
    assert _lib.wait_timeout_flags(DEV) == 0


def test_bands_of_a_slab_equal_the_whole_image():
    from sapa_b200 import sharding
    from sapa_b200.functions import fused_forward_raw
    B, d, C, H, W, r = 2, 40, 300, 60, 64, 2
    q, k, v = _rand(1, B, d, 2 * H, 2 * W, scale=0.5), _rand(2, B, d, H, W, scale=0.5), _rand(3, B, C, H, W)
    whole = fused_forward_raw(q, k, v, 5, 2, False)[0]
    lo, rows = 11, 40
    slab = sharding.RowSlab(B, d, C, rows, W, torch.float32, torch.device(DEV), 5, 2)
    slab.key_padded.copy_(k[:, :, lo - r:lo + rows + r])
    slab.value_padded.copy_(v[:, :, lo - r:lo + rows + r])
    hi = slice(2 * lo, 2 * (lo + rows))
    ql, out = q[:, :, hi].contiguous(), torch.empty(B, C, 2 * rows, 2 * W, device=DEV)
    for begin, end in ((0, 4), (4, rows - 3), (rows - 3, rows)):
        slab._launch(ql, out, begin, end)
    assert torch.equal(out, whole[:, :, hi])


@pytest.mark.parametrize("shape", [(1, 64, 250, 96, 96), (2, 16, 64, 40, 96), (2, 16, 140, 40, 96)], ids=lambda s: "B%d_d%d_C%d_%dx%d" % s)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_slab_goes_the_way_of_its_image(shape, dtype):
    """The output and the query gradient of a few rows equal those of the whole image bit for bit, also where the rows alone are a small
    problem, and the output of an image by itself that in its batch."""
    import sapa_b200 as sp
    from sapa_b200 import sharding
    B, d, C, H, W = shape
    q, k, v = (x.to(dtype) for x in (_rand(1, B, d, 2 * H, 2 * W, scale=0.5), _rand(2, B, d, H, W, scale=0.5), _rand(3, B, C, H, W)))
    go = _rand(4, B, C, 2 * H, 2 * W).to(dtype)
    t = [x.clone().requires_grad_() for x in (q, k, v)]
    whole = sp.sapa_fused(*t, 5, 2)
    gq = torch.autograd.grad(whole, t, go)[0]
    assert torch.equal(sp.sapa_fused(*(x[-1:] for x in (q, k, v)), 5, 2)[0], whole.detach()[-1])
    r, rows = 2, 8
    for lo in (2, 13):
        hi = slice(2 * lo, 2 * (lo + rows))
        slab = sharding.RowSlab(B, d, C, rows, W, dtype, torch.device(DEV), 5, 2)
        slab.key_padded.copy_(k[:, :, lo - r:lo + rows + r])
        slab.value_padded.copy_(v[:, :, lo - r:lo + rows + r])
        ql, out = q[:, :, hi].contiguous(), torch.empty(B, C, 2 * rows, 2 * W, dtype=dtype, device=DEV)
        slab._launch(ql, out, 0, rows)
        assert torch.equal(out, whole.detach()[:, :, hi])
        slab.attn = torch.empty(B, 25, 2 * rows, 2 * W, dtype=dtype, device=DEV)
        slab._launch(ql, out, 0, rows)
        assert torch.equal(out, whole.detach()[:, :, hi])
        assert torch.equal(slab.backward(go[:, :, hi].contiguous(), ql)[0], gq[:, :, hi])


# sums of numbers of one sign, as behind a ReLU: every accumulation of a product in tensor memory rounds the whole sum down.  64 channels are 24 of them, half an
# ulp (6e-8) of a sum that has grown to half on average: 7e-7, and 9.8e-7 measured; the sums of products round to nearest
@pytest.mark.parametrize("channels", [64, 100, 256, 720])
def test_features_of_one_sign(channels):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, H, W = 2, 48, 64
    hi, lo = _rand(1, B, channels, 2 * H, 2 * W).abs() + 0.25, _rand(2, B, channels, H, W).abs() + 0.25
    want = torch.stack([(hi.double() * w).sum(1) for w in _windows(lo.double())], 1)
    inside = want != 0

    def off(got):
        return float(((got.double() - want)[inside] / want[inside]).abs().mean())
    assert off(sp.qk(hi, lo, 5, 2)) < 1.3e-6
    assert _lib.last_kernels() == ["sapa_strip_sim_kernel<logits>"]
    # the same sums in stage 1 of the backward: logit gradients of a uniform map are (dA - mean dA) / 25
    attn = torch.full((B, 25, 2 * H, 2 * W), 0.04, device=DEV).requires_grad_()
    got = torch.autograd.grad(sp.av(attn, lo, 5, 2), attn, hi)[0]
    assert off(got) < 1.3e-6
