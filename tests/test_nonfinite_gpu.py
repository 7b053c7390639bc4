"""Rows that are not multiples of 16 bytes, and gradients gathered on 4 x 32 tiles, in 16 bits: an infinity or a NaN reaches the pixels
(cells) whose window holds it and no other, as in sums over the window alone - the tensor-core kernels multiply whole fragments,
with weights of zero beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
INF, NAN = float("inf"), float("nan")

# (image, channel, row, column, value) of a low-resolution tensor: inside a tile, at its edges and at the image's, two of one window
SPOTS = [(0, 3, 7, 9, INF), (0, 5, 11, 15, NAN), (1, 0, 0, 0, -INF), (1, 7, 12, 16, INF), (1, 7, 13, 17, INF), (1, 9, 5, 24, INF)]


def _rand(*shape, scale=1.0, dtype):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(sum(shape))) * scale).to(dtype).to(DEV)


def _planted(t):
    bad = t.clone()
    for n, c, y, x, v in SPOTS:
        bad[n, c, y, x] = v
    return bad


def _near(mask):
    """Low-resolution cells with a marked one in their 5 x 5 neighbourhood."""
    return torch.nn.functional.max_pool2d(mask.float(), 5, 1, 2) > 0


def _up(mask):
    return mask.repeat_interleave(2, 2).repeat_interleave(2, 3)


def _same_elsewhere(got, clean, reached, dtype):
    """Where nothing reaches, the result of the clean input (sums in another order, one rounding: two ulps); where something does, no
    finite number."""
    assert not torch.isfinite(got[reached]).any()
    a, b = got[~reached].float(), clean[~reached].float()
    assert bool(((a - b).abs() <= 2 * torch.finfo(dtype).eps * b.abs() + 1e-6 * float(b.abs().max())).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("W", [25, 42])
def test_values(W, dtype):
    import sapa_b200 as sp
    H, C = 17, 40
    value = _rand(2, C, H, W, dtype=dtype)
    bad = _planted(value)
    attn = (torch.rand(2, 25, 2 * H, 2 * W, generator=torch.Generator().manual_seed(1)) + 0.1).to(dtype).to(DEV)
    reached = _up(_near(~torch.isfinite(bad)))
    got = sp.av(attn, bad, 5, 2)
    _same_elsewhere(got, sp.av(attn, value, 5, 2), reached, dtype)
    only_inf = _up(_near(bad == INF) & ~_near((bad != bad) | (bad == -INF)))
    assert bool((got[only_inf] == INF).all())
    if W % 2:      # the fused kernel of odd rows: weights in two terms of both signs, some below the smallest 16-bit number
        for scale in (0.5, 3.0):
            q, k = _rand(2, 8, 2 * H, 2 * W, scale=scale, dtype=dtype), _rand(2, 8, H, W, scale=scale, dtype=dtype)
            got = sp.sapa_fused(q, k, bad, 5, 2)
            _same_elsewhere(got, sp.sapa_fused(q, k, value, 5, 2), reached, dtype)
            assert bool((got[only_inf] == INF).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("W", [25, 42])
def test_query_gradient(W, dtype):
    """Stage 1 of the backward: its query gradient, with infinities among the values."""
    import sapa_b200 as sp
    H, C = 17, 40
    q, k, value = (_rand(*s, dtype=dtype) for s in ((2, 8, 2 * H, 2 * W), (2, 8, H, W), (2, C, H, W)))
    go = _rand(2, C, 2 * H, 2 * W, dtype=dtype)
    bad = _planted(value)
    reached = _up(_near(~torch.isfinite(bad))).any(1, keepdim=True).expand(-1, 8, -1, -1)

    def grad(v):
        t = q.clone().requires_grad_()
        return torch.autograd.grad(sp.sapa_fused(t, k, v, 5, 2), t, go)[0]
    _same_elsewhere(grad(bad), grad(value), reached, dtype)
    # the separate op: logit gradients are given, keys hold the infinities
    ds = _rand(2, 25, 2 * H, 2 * W, dtype=dtype)
    key = _rand(2, 40, H, W, dtype=dtype)

    def grad_qk(kk):
        t = _rand(2, 40, 2 * H, 2 * W, dtype=dtype).requires_grad_()
        return torch.autograd.grad(sp.qk(t, kk, 5, 2), t, ds)[0]
    _same_elsewhere(grad_qk(_planted(key)), grad_qk(key), _up(_near(~torch.isfinite(_planted(key)))), dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("W", [25, 42, 64])      # 64: tiles of 4 x 32 cells, whose fragments are wider than a tile's reach
def test_gathered_gradients(W, dtype):
    """Value gradient of av and key gradient of qk, with infinities among the high-resolution gradients (queries)."""
    import sapa_b200 as sp
    H, C = 17, 40
    hi = _rand(2, C, 2 * H, 2 * W, dtype=dtype)
    bad = hi.clone()
    for n, c, y, x, v in SPOTS:
        bad[n, c, 2 * y + x % 2, 2 * x + y % 2] = v
    bad[0, 8, 16, 21] = INF      # a pixel that the next tile's fragments hold beside those that reach it
    marked = ~torch.isfinite(bad)
    reached = _near(torch.nn.functional.max_pool2d(marked.float(), 2) > 0)
    slots = (torch.rand(2, 25, 2 * H, 2 * W, generator=torch.Generator().manual_seed(1)) + 0.1).to(dtype).to(DEV)
    low = _rand(2, C, H, W, dtype=dtype)

    def value_grad(go):
        t = low.clone().requires_grad_()
        return torch.autograd.grad(sp.av(slots, t, 5, 2), t, go)[0]

    def key_grad(q):
        t = low.clone().requires_grad_()
        return torch.autograd.grad(sp.qk(q, t, 5, 2), t, slots)[0]
    for grad in (value_grad, key_grad):
        _same_elsewhere(grad(bad), grad(hi), reached, dtype)


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.bfloat16, 2e-2), (torch.float16, 4e-3)])
@pytest.mark.parametrize("points", [9, 1, 4, 16])      # the unrolled form and the one for any number
def test_sampling_offsets(points, dtype, tol):
    """A sampling point at an infinite or undefined place lies outside the image: logit 0, nothing added to the output, no gradient.
    tol: 2-norm against the float64 ops, as in test_outlier_lists_gpu.py."""
    import sapa_b200 as sp
    B, C, d, H, W, G = 2, 24, 8, 9, 16, 2
    q, k, v, o, go = (torch.randn(*s, generator=torch.Generator().manual_seed(i)) * f for i, (s, f) in enumerate((
        ((B, d, 2 * H, 2 * W), 0.5), ((B, d, H, W), 0.5), ((B, C, H, W), 1.0), ((B, 2 * points * G, 2 * H, 2 * W), 0.6), ((B, C, 2 * H, 2 * W), 1.0))))
    o = (o * 64).round() / 64 + 1 / 128      # positions are exact in float32: the same cells as in float64
    for n, (c, y, x, value) in enumerate(((0, 0, 0, INF), (1, 3, 5, NAN), (2 * points, 7, 31, -INF), (0, 4, 4, NAN), (2 * points - 1, 17, 12, INF), (1, 8, 8, -INF))):
        o[n % B, c, y, x] = value
    o[0, :, 11, 20] = INF      # every point of a pixel
    t = [x.to(dtype).to(DEV).requires_grad_() for x in (q, k, v, o)]
    r = [x.detach().double().requires_grad_() for x in t]
    a = torch.rand(B, G, points, 2 * H, 2 * W, generator=torch.Generator().manual_seed(9)).to(dtype).to(DEV).requires_grad_()
    ra, up = a.detach().double().requires_grad_(), go.to(dtype).to(DEV)

    def results(x, attn, g):
        fused, logits, out = sp.deform_sapa_fused(*x, points, 2, G), sp.deform_qk(x[0], x[1], x[3], points, 2, G), sp.deform_av(attn, x[2], x[3], points, 2, G)
        return [fused, logits, out, *torch.autograd.grad(fused, x, g), *torch.autograd.grad(logits, [x[0], x[1], x[3]], attn.detach()),
                *torch.autograd.grad(out, [attn, x[2], x[3]], g)]
    for n, (x, y) in enumerate(zip(results(t, a, up), results(r, ra, up.double()))):
        error, norm = float((x.detach().double() - y.detach()).norm()), float(y.detach().norm())
        assert error <= tol * (norm or 1.0), n      # one point: its attention is 1, its logit has no gradient
