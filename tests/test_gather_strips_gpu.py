"""The gather kernel that walks strips of columns down the image (value and key gradients of larger problems): partial strips and blocks
of 128 channels, output rows that outnumber its ring, several items a CTA, rows of neighbouring slabs, infinities."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INF, NAN = float("inf"), float("nan")


def _rand(seed, *shape, dtype):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).to(DEV)


def _gather(go, wt, halo=0):
    """G[c][u] = sum of go[c][p] wt[k][p] over the pixels and slots with win_k(p) = u, in float64; with `halo` rows around the image."""
    (B, C, sH, sW), H, W = go.shape, go.shape[2] // 2, go.shape[3] // 2
    out = torch.zeros(B, C, H + 4, W + 4, dtype=torch.float64, device=go.device)
    for k in range(25):
        out[:, :, k // 5:k // 5 + H, k % 5:k % 5 + W] += (go.double() * wt[:, k:k + 1].double()).view(B, C, H, 2, W, 2).sum((3, 5))
    return out[:, :, 2 - halo:2 + halo + H, 2:-2]


def _value_grad(go, wt, C, H, W):
    import sapa_b200 as sp
    v = torch.zeros(go.shape[0], C, H, W, dtype=go.dtype, device=DEV, requires_grad=True)
    return torch.autograd.grad(sp.av(wt, v, 5, 2), v, go)[0]


# 2-norms.  float32: three-term tf32 products (1e-7) and about twenty roundings of a sum (5e-7 measured, 5.3e-7 on the tiles).  16 bits:
# exact products, float32 sums, one rounding of the result (half an ulp at most, 0.3 of one in the mean)
TOLERANCE = [(torch.float32, 6e-7), (torch.bfloat16, 2e-3), (torch.float16, 2.5e-4)]


@pytest.mark.parametrize("dtype,tol", TOLERANCE)
@pytest.mark.parametrize("shape", [(1, 600, 28, 72), (6, 129, 70, 40), (40, 128, 20, 16), (2, 256, 150, 104), (40, 128, 24, 32)], ids=lambda s: "B%d_C%d_%dx%d" % s)
def test_strips_vs_float64(shape, dtype, tol):
    from sapa_b200 import _lib
    B, C, H, W = shape
    wt = torch.softmax(_rand(1, B, 25, 2 * H, 2 * W, dtype=torch.float32), 1).to(dtype)
    go = _rand(2, B, C, 2 * H, 2 * W, dtype=dtype)
    want = _gather(go, wt)
    for _ in range(3):
        got = _value_grad(go, wt, C, H, W)
        assert _lib.last_kernels()[-1] == "sapa_gath_umma_kernel" or W == 16      # the smallest images are left to the tiles
        assert float((got.double() - want).norm() / want.norm()) < tol
        assert float((got.double() - want).abs().max() / want.abs().max()) < 4 * tol
    assert _lib.wait_timeout_flags(DEV) == 0


@pytest.mark.parametrize("dtype,tol", TOLERANCE)
def test_strips_of_a_slab(dtype, tol):
    """The gradients of a slab's neighbour rows, which its pixels reach."""
    from sapa_b200 import _lib, sharding
    B, d, C, H, W, r = 2, 300, 520, 20, 80, 2
    code = _lib.dtype_code(torch.empty(0, dtype=dtype))
    slab = sharding.RowSlab(B, d, C, H, W, dtype, torch.device(DEV), 5, 2)
    slab.key_padded.copy_(_rand(1, B, d, H + 2 * r, W, dtype=dtype) * 0.1)
    slab.value_padded.copy_(_rand(2, B, C, H + 2 * r, W, dtype=dtype))
    q, go = _rand(3, B, d, 2 * H, 2 * W, dtype=dtype) * 0.5, _rand(4, B, C, 2 * H, 2 * W, dtype=dtype)
    slab.forward(q, keep_attn=True)
    mq, mk, mv = torch.empty_like(q), torch.empty_like(slab.key_padded), torch.empty_like(slab.value_padded)
    nb = _lib.fused_backward_workspace(B, H, W, 5, 2, code)
    ws = torch.empty(nb, dtype=torch.uint8, device=DEV)
    _lib.call("sapa_fused_backward_slab", torch.device(DEV), go, q, slab.key_padded, slab.value_padded, slab.attn, mq, mk, mv, ws, nb,
              B, d, C, H, W, r, r, 5, 2, code)
    assert _lib.last_kernels()[-2:] == ["sapa_gath_umma_kernel"] * 2
    ds = ws[:B * 25 * 4 * H * W * q.element_size()].view(dtype).view(B, 25, 2 * H, 2 * W)
    for got, want in ((mv, _gather(go, slab.attn, r)), (mk, _gather(q, ds, r))):
        assert got.shape == want.shape and float((got.double() - want).norm() / want.norm()) < tol
    assert _lib.wait_timeout_flags(DEV) == 0


@pytest.mark.parametrize("dtype,tol", TOLERANCE)
def test_strips_keep_infinities_to_their_cells(dtype, tol):
    from sapa_b200 import _lib
    B, C, H, W = 2, 300, 40, 72
    wt = (torch.rand(B, 25, 2 * H, 2 * W, generator=torch.Generator().manual_seed(1)) + 0.1).to(dtype).to(DEV)
    go = _rand(2, B, C, 2 * H, 2 * W, dtype=dtype)
    bad = go.clone()
    for n, c, y, x, v in ((0, 3, 0, 0, INF), (0, 130, 41, 63, NAN), (1, 299, 79, 143, -INF), (1, 7, 33, 64, INF), (1, 7, 35, 70, INF)):
        bad[n, c, y, x] = v
    marked = F.max_pool2d((~torch.isfinite(bad)).float(), 2) > 0
    reached = F.max_pool2d(marked.float(), 5, 1, 2) > 0
    clean, got = _value_grad(go, wt, C, H, W), _value_grad(bad, wt, C, H, W)
    assert _lib.last_kernels()[-1] == "sapa_gath_umma_kernel"
    assert not torch.isfinite(got[reached]).any()
    a, b = got[~reached].double(), clean[~reached].double()
    assert float((a - b).abs().max() / b.abs().max()) < 4 * tol      # cells of the marked rows: sums in another order
    only = F.max_pool2d(F.max_pool2d((bad == INF).float(), 2), 5, 1, 2) > 0
    only &= ~(F.max_pool2d(F.max_pool2d(((bad != bad) | (bad == -INF)).float(), 2), 5, 1, 2) > 0)
    assert bool((got[only] == INF).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("top,bottom", [(40, 2), (3, 45)])
def test_rows_that_no_pixel_reaches(top, bottom, dtype):
    """A slab's gradients in a frame with more rows around it than its pixels reach: some items of a CTA have none, others have a NaN."""
    from sapa_b200 import _lib
    B, C, H, W = 75, 64, 30, 32
    code = _lib.dtype_code(torch.empty(0, dtype=dtype))
    q, k = _rand(1, B, C, 2 * H, 2 * W, dtype=dtype), _rand(2, B, C, top + H + bottom, W, dtype=dtype)
    go, v = _rand(3, B, C, 2 * H, 2 * W, dtype=dtype), _rand(4, B, C, top + H + bottom, W, dtype=dtype)
    attn = torch.softmax(_rand(5, B, 25, 2 * H, 2 * W, dtype=torch.float32), 1).to(dtype)
    marked = torch.zeros(B, C, top + H + bottom, W, device=DEV)
    for n in range(0, B, 4):
        for c, y, x in ((n % C, 0, 2 * (n % W)), (7, 2 * H - 1, 5), (9, 31, 40)):
            go[n, c, y, x] = NAN
            marked[n, c, top + y // 2, x // 2] = 1
    reached = F.max_pool2d(marked, 5, 1, 2) > 0
    gq, gk, gv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    nb = _lib.fused_backward_workspace(B, H, W, 5, 2, code)
    _lib.call("sapa_fused_backward_slab", torch.device(DEV), go, q, k, v, attn, gq, gk, gv, torch.empty(nb, dtype=torch.uint8, device=DEV), nb, B, C, C, H, W,
              top, bottom, 5, 2, code)
    assert _lib.last_kernels()[-1] == "sapa_gath_umma_kernel"
    assert torch.equal(~torch.isfinite(gv), reached)
    outside = torch.ones(top + H + bottom, dtype=torch.bool, device=DEV)
    outside[top - 2:top + H + 2] = False
    assert not gv[:, :, outside].any()
    assert _lib.wait_timeout_flags(DEV) == 0
