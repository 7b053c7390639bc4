"""The 16-bit fused forward on strips of columns, both products on the 5th-generation tensor cores: every count of query channels up to
its limit and beyond, partial strips and blocks of 128 channels, rows that outnumber its rings, bands of rows, the attention map."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INF, NAN = float("inf"), float("nan")


def _rand(seed, *shape, dtype, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype).to(DEV)


def _forward(q, k, v):
    H, W = v.shape[2:]

    def window(t):
        padded = F.pad(t.double(), (2, 2, 2, 2))
        return [padded[:, :, i // 5:i // 5 + H, i % 5:i % 5 + W].repeat_interleave(2, 2).repeat_interleave(2, 3) for i in range(25)]
    attn = torch.softmax(torch.stack([(q.double() * w).sum(1) for w in window(k)], 1), 1)
    return sum(attn[:, i:i + 1] * w for i, w in enumerate(window(v))), attn


# 2-norms.  The attention map is rounded once (half an ulp at most, 0.3 of one in the mean: 1.7e-3 in bfloat16, 2.1e-4 in float16), the
# output is a sum of products with rounded weights, rounded again (1.4 of that)
@pytest.mark.parametrize("dtype,tol", [(torch.bfloat16, 2.1e-3), (torch.float16, 2.6e-4)])
@pytest.mark.parametrize("shape", [(1, 24, 8, 3, 16), (1, 24, 8, 53, 16), (2, 130, 16, 7, 40), (3, 300, 24, 41, 72), (40, 48, 33, 20, 24), (2, 256, 48, 150, 104), (5, 200, 64, 70, 136),
                                   (1, 64, 65, 9, 32), (2, 64, 1, 12, 48)], ids=lambda s: "B%d_C%d_d%d_%dx%d" % s)
def test_strips_vs_float64(shape, dtype, tol):
    from sapa_b200 import _lib
    from sapa_b200.functions import fused_forward_raw
    B, C, d, H, W = shape
    q, k, v = _rand(1, B, d, 2 * H, 2 * W, dtype=dtype, scale=0.5), _rand(2, B, d, H, W, dtype=dtype, scale=0.5), _rand(3, B, C, H, W, dtype=dtype)
    want, want_attn = _forward(q, k, v)
    first = None
    for keep in (False, True, True):
        out, attn = fused_forward_raw(q, k, v, 5, 2, keep)
        # the smallest image, and more than 64 query channels, are left to the tiles
        assert _lib.last_kernels() == ["sapa_strip_fwd_kernel"] or d > 64 or C * H * W < 2e4
        assert float((out.double() - want).norm() / want.norm()) < 1.4 * tol
        assert float((out.double() - want).abs().max() / want.abs().max()) < 4 * tol
        assert first is None or torch.equal(out, first)
        first = out
    assert float((attn.double() - want_attn).norm() / want_attn.norm()) < tol
    one = fused_forward_raw(*(t[-1:].contiguous() for t in (q, k, v)), 5, 2, False)[0]
    assert torch.equal(one[0], first[-1])            # images are independent
    assert _lib.wait_timeout_flags(DEV) == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_bands_of_a_slab(dtype):
    """Rows of a padded slab, computed in bands, equal the rows of the whole image bit for bit."""
    from sapa_b200 import sharding
    from sapa_b200.functions import fused_forward_raw
    B, d, C, H, W, r = 2, 40, 136, 40, 56, 2
    q, k, v = _rand(1, B, d, 2 * H, 2 * W, dtype=dtype, scale=0.5), _rand(2, B, d, H, W, dtype=dtype, scale=0.5), _rand(3, B, C, H, W, dtype=dtype)
    whole = fused_forward_raw(q, k, v, 5, 2, False)[0]
    lo, rows = 12, 20
    slab = sharding.RowSlab(B, d, C, rows, W, dtype, torch.device(DEV), 5, 2)
    slab.key_padded.copy_(k[:, :, lo - r:lo + rows + r])
    slab.value_padded.copy_(v[:, :, lo - r:lo + rows + r])
    hi = slice(2 * lo, 2 * (lo + rows))
    ql, out = q[:, :, hi].contiguous(), torch.empty(B, C, 2 * rows, 2 * W, dtype=dtype, device=DEV)
    for begin, end in ((0, 4), (4, rows - 3), (rows - 3, rows)):
        slab._launch(ql, out, begin, end)
    assert torch.equal(out, whole[:, :, hi])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(2, 300, 24, 40, 72), (1, 160, 64, 9, 16), (2, 136, 40, 14, 40)], ids=lambda s: "B%d_C%d_d%d_%dx%d" % s)
def test_strips_keep_infinities_to_their_windows(shape, dtype):
    """An infinity or NaN of the value reaches the pixels whose window holds it, and those get what their weights make of it; every
    other output has the bits that it has without it."""
    from sapa_b200 import _lib
    from sapa_b200.functions import fused_forward_raw
    B, C, d, H, W = shape
    q, k, v = _rand(1, B, d, 2 * H, 2 * W, dtype=dtype, scale=0.5), _rand(2, B, d, H, W, dtype=dtype, scale=0.5), _rand(3, B, C, H, W, dtype=dtype)
    bad = v.clone()
    for n, c, y, x, what in ((0, 3, 0, 0, INF), (0, C - 1, 7, 11, NAN), (B - 1, C - 1, H - 1, W - 1, -INF), (B - 1, 7, 5, 14, INF), (B - 1, 7, 6, 15, INF),
                             (0, 20, 4, 9, INF), (0, 20, 6, 10, -INF), (0, 21, 3, 8, INF), (0, 21, 4, 8, NAN)):
        bad[n, c, y, x] = what
    for keep in (False, True):
        clean, got = fused_forward_raw(q, k, v, 5, 2, keep)[0], fused_forward_raw(q, k, bad, 5, 2, keep)[0]
        attn = fused_forward_raw(q, k, bad, 5, 2, True)[1]
        assert _lib.last_kernels() == ["sapa_strip_fwd_kernel"]
        assert torch.isfinite(attn).all()
        reached = (F.max_pool2d((~torch.isfinite(bad)).float(), 5, 1, 2) > 0).repeat_interleave(2, 2).repeat_interleave(2, 3)
        assert torch.equal(got[~reached], clean[~reached])
        want = torch.zeros(B, C, 2 * H, 2 * W, dtype=torch.float64, device=DEV)
        padded = F.pad(bad.double(), (2, 2, 2, 2))
        for i in range(25):
            window = padded[:, :, i // 5:i // 5 + H, i % 5:i % 5 + W].repeat_interleave(2, 2).repeat_interleave(2, 3)
            want += attn[:, i:i + 1].double() * window
        assert not torch.isfinite(want[reached]).any()
        a, b = got[reached].double(), want[reached]
        assert bool(((a == b) | (torch.isnan(a) & torch.isnan(b))).all())
    assert _lib.wait_timeout_flags(DEV) == 0
