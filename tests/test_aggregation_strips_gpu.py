"""The aggregation kernel that walks strips of columns down the image: partial strips and blocks of 128 channels, more rows than its ring in
tensor memory, several items a CTA, padded slabs, infinities."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INF, NAN = float("inf"), float("nan")

# 2-norms.  float32: three-term tf32 products (1e-7) and about eight roundings of a sum (4.7e-7 measured, 6.9e-7 on the tiles).  16 bits:
# exact products, float32 sums, one rounding of the result (half an ulp at most, 0.3 of one in the mean)
TOLERANCE = [(torch.float32, 6e-7), (torch.bfloat16, 2e-3), (torch.float16, 2.5e-4)]


def _rand(seed, *shape, dtype):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).to(DEV)


def _aggregate(wt, value):
    """out[c, p] = sum_k wt[k, p] window_k(value)[c, p] in float64."""
    H, W = value.shape[2:]
    padded = F.pad(value.double(), (2, 2, 2, 2))
    return sum(wt[:, k:k + 1].double() * padded[:, :, k // 5:k // 5 + H, k % 5:k % 5 + W].repeat_interleave(2, 2).repeat_interleave(2, 3)
               for k in range(25))


@pytest.mark.parametrize("dtype,tol", TOLERANCE)
@pytest.mark.parametrize("shape", [(2, 600, 88, 72), (6, 200, 70, 40), (40, 128, 20, 16), (2, 256, 150, 104), (3, 48, 130, 200), (40, 128, 30, 16)],
                         ids=lambda s: "B%d_C%d_%dx%d" % s)
def test_strips_vs_float64(shape, dtype, tol):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, C, H, W = shape
    wt = torch.softmax(_rand(1, B, 25, 2 * H, 2 * W, dtype=torch.float32), 1).to(dtype)
    value = _rand(2, B, C, H, W, dtype=dtype)
    want = _aggregate(wt, value)
    for _ in range(3):
        got = sp.av(wt, value, 5, 2)
        # the smallest images are left to the tiles in 16 bits
        assert _lib.last_kernels() == ["sapa_strip_kernel"] or (dtype != torch.float32 and C * H * W < 6e4 and W == 16)
        assert float((got.double() - want).norm() / want.norm()) < tol
        assert float((got.double() - want).abs().max() / want.abs().max()) < 4 * tol
    assert _lib.wait_timeout_flags(DEV) == 0


@pytest.mark.parametrize("dtype,tol", TOLERANCE)
def test_strips_of_a_padded_slab(dtype, tol):
    """SAPA-D on a slab with neighbour rows above and below: its aggregation reads a value tensor with more rows than its pixels have."""
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, C, d, H, W, G, P = 2, 384, 32, 48, 64, 4, 9
    q, k, v = (_rand(i, *s, dtype=dtype) * f for i, (s, f) in enumerate((((B, d, 2 * H, 2 * W), 0.5), ((B, d, H, W), 0.5), ((B, C, H, W), 1.0))))
    off = _rand(4, B, 2 * G * P, 2 * H, 2 * W, dtype=dtype).clamp(-3, 3) * 0.4
    whole = sp.deform_sapa_fused(q, k, v, off, P, 2, G)
    top, halo, rows = 8, 3, 28                        # rows 8 .. 35 with three neighbours each
    hi, lo = slice(2 * top, 2 * (top + rows)), slice(top - halo, top + rows + halo)
    code = _lib.dtype_code(q)
    nbytes = int(_lib.lib().sapa_deform_fused_forward_workspace(B, rows, W, P, 2, G, code))
    ws, out = torch.empty(nbytes, dtype=torch.uint8, device=DEV), torch.empty(B, C, 2 * rows, 2 * W, dtype=dtype, device=DEV)
    _lib.call("sapa_deform_fused_forward_slab", q.device, *(t.contiguous() for t in (q[:, :, hi], k[:, :, lo], v[:, :, lo], off[:, :, hi])), out, None,
              ws, nbytes, B, d, C, rows, W, halo, halo, P, 2, G, code)
    assert "sapa_strip_kernel" in _lib.last_kernels()
    want = whole[:, :, hi].double()
    assert float((out.double() - want).norm() / want.norm()) < 4 * tol
    assert _lib.wait_timeout_flags(DEV) == 0


@pytest.mark.parametrize("dtype,tol", TOLERANCE)
def test_strips_keep_infinities_to_their_pixels(dtype, tol):
    import sapa_b200 as sp
    from sapa_b200 import _lib
    B, C, H, W = 3, 300, 40, 72
    wt = (torch.rand(B, 25, 2 * H, 2 * W, generator=torch.Generator().manual_seed(1)) + 0.1).to(dtype).to(DEV)
    value = _rand(2, B, C, H, W, dtype=dtype)
    bad = value.clone()
    for n, c, y, x, v in ((0, 3, 0, 0, INF), (0, 130, 20, 31, NAN), (1, 299, 39, 71, -INF), (2, 7, 16, 32, INF), (2, 7, 17, 35, INF)):
        bad[n, c, y, x] = v

    def near(mask):
        return (F.max_pool2d(mask.float(), 5, 1, 2) > 0).repeat_interleave(2, 2).repeat_interleave(2, 3)
    reached = near(~torch.isfinite(bad))
    clean, got = sp.av(wt, value, 5, 2), sp.av(wt, bad, 5, 2)
    assert _lib.last_kernels() == ["sapa_strip_kernel"]
    assert not torch.isfinite(got[reached]).any()
    a, b = got[~reached].double(), clean[~reached].double()
    assert float((a - b).abs().max() / b.abs().max()) < 4 * tol      # pixels of the marked rows: sums in another order
    only = near(bad == INF) & ~near((bad != bad) | (bad == -INF))
    assert bool((got[only] == INF).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_strips_with_infinite_weights_and_values(dtype):
    """Weights that are not finite touch their own pixel; all results are those of the sum over the window's cells inside the image."""
    import sapa_b200 as sp
    B, C, H, W = 3, 300, 40, 72
    wt = torch.randn(B, 25, 2 * H, 2 * W, generator=torch.Generator().manual_seed(1)).to(dtype).to(DEV)      # of both signs
    value = _rand(2, B, C, H, W, dtype=dtype)
    clean = sp.av(wt, value, 5, 2)
    wt[0, 3, 20, 20], wt[0, 12, 0, 0], wt[1, 24, 79, 143], wt[2, :, 11, 64] = INF, NAN, -INF, NAN
    wt[1, 7, 30:34, 60:70] = 0
    for n, c, y, x, v in ((0, 3, 9, 9, INF), (0, 130, 20, 31, NAN), (1, 7, 16, 32, INF), (1, 7, 17, 35, -INF), (1, 8, 15, 32, -INF), (2, 9, 5, 31, INF)):
        value[n, c, y, x] = v
    value[1, 200] = INF
    value[2, 100] = NAN
    inside = F.pad(torch.ones(1, 1, H, W, device=DEV), (2, 2, 2, 2))
    padded, want = F.pad(value.double(), (2, 2, 2, 2)), torch.zeros(B, C, 2 * H, 2 * W, dtype=torch.float64, device=DEV)
    for k in range(25):
        at = (slice(None), slice(None), slice(k // 5, k // 5 + H), slice(k % 5, k % 5 + W))
        term = wt[:, k:k + 1].double() * padded[at].repeat_interleave(2, 2).repeat_interleave(2, 3)
        want += torch.where(inside[at].repeat_interleave(2, 2).repeat_interleave(2, 3) > 0, term, torch.zeros_like(term))
    got = sp.av(wt, value, 5, 2)
    odd = ~torch.isfinite(want)
    a, b = got[odd].double(), want[odd]
    assert bool(((a == b) | (torch.isnan(a) & torch.isnan(b))).all())
    same = F.max_pool2d((~torch.isfinite(value)).float(), 5, 1, 2).repeat_interleave(2, 2).repeat_interleave(2, 3) == 0
    assert torch.isfinite(got[~odd]).all()
    untouched = same & (torch.isfinite(wt).all(1, keepdim=True)) & (wt[:, 7:8] != 0)
    assert torch.equal(got[untouched], clean[untouched])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_what_is_not_finite_costs_little(dtype):
    """A NaN in an input, or nothing else in it, does not take the kernels on strips hundreds of times as long (measured on 8 x 256 x 64x64: one NaN 1.6
    to 3.3 times, nothing else 5 to 12; all outputs formed one by one 130 to 350)."""
    import sapa_b200 as sp
    B, C, H, W = 4, 256, 64, 64
    wt = torch.softmax(_rand(1, B, 25, 2 * H, 2 * W, dtype=torch.float32), 1).to(dtype)
    value, go = _rand(2, B, C, H, W, dtype=dtype), _rand(3, B, C, 2 * H, 2 * W, dtype=dtype)

    def time(a, v, g):
        a, v = a.clone().requires_grad_(), v.clone().requires_grad_()
        out, best = sp.av(a, v, 5, 2), float("inf")
        for _ in range(6):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            torch.cuda._sleep(200000)                 # the calls are queued before the first one starts
            e[0].record()
            with torch.no_grad():
                sp.av(a, v, 5, 2)
            torch.autograd.grad(out, (a, v), g, retain_graph=True)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]))
        return best
    one_v, one_g = value.clone(), go.clone()
    one_v[1, 3, 20, 20] = one_g[1, 3, 40, 40] = NAN
    finite = time(wt, value, go)
    assert time(wt, one_v, one_g) < 10 * finite
    assert time(wt, torch.full_like(value, NAN), torch.full_like(go, NAN)) < 40 * finite
    assert time(torch.full_like(wt, NAN), value, go) < 40 * finite
