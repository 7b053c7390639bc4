"""An image's results have the same bits whatever batch it is in: the choice between kernels sees one image.  Except the aggregation by itself in
float32, whose choice sees the whole problem: equal to rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
B = 20

# channels of value and query, rows, columns: on both sides of the lines between tiles and strips, and where a batch of them is a large problem
SHAPES = [(64, 32, 32, 32), (128, 64, 24, 40), (32, 16, 64, 64), (256, 64, 16, 16), (128, 16, 48, 48), (64, 32, 128, 16), (128, 64, 64, 64)]


def _rand(seed, *shape, dtype, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype).to(DEV)


def _equal(a, b, rounding):
    """rounding: two kernels' sums of 25 products in float32, 7e-7 each from float64"""
    return torch.equal(a, b) if not rounding else float((a.double() - b.double()).norm()) <= 1.4e-6 * float(b.double().norm())


def _results(t, up, ops):
    t = [x.clone().requires_grad_() for x in t]
    out = ops(*t)
    return [out.detach(), *torch.autograd.grad(out, t, up)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "C%d_d%d_%dx%d" % s)
def test_window_ops(shape, dtype):
    import sapa_b200 as sp
    C, d, H, W = shape
    q, k, v = _rand(1, B, d, 2 * H, 2 * W, dtype=dtype, scale=0.5), _rand(2, B, d, H, W, dtype=dtype, scale=0.5), _rand(3, B, C, H, W, dtype=dtype)
    go, attn = _rand(4, B, C, 2 * H, 2 * W, dtype=dtype), torch.softmax(_rand(5, B, 25, 2 * H, 2 * W, dtype=torch.float32), 1).to(dtype)
    # with each op, which of its results (the output, then the gradients) is the aggregation by itself
    for t, up, op, agg in (((q, k, v), go, lambda *x: sp.sapa_fused(*x, 5, 2), None), ((q, k), attn, lambda *x: sp.qk(*x, 5, 2), 1),
                           ((attn, v), go, lambda *x: sp.av(*x, 5, 2), 0)):
        batch = _results(t, up, op)
        for n in (0, B - 1):
            for i, (a, b) in enumerate(zip(batch, _results([x[n:n + 1] for x in t], up[n:n + 1], op))):
                assert _equal(a[n:n + 1], b, i == agg and dtype == torch.float32), (i, agg)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(128, 32, 32, 32), (256, 64, 24, 40), (64, 64, 64, 64)], ids=lambda s: "C%d_d%d_%dx%d" % s)
def test_sampled_ops(shape, dtype):
    """SAPA-D with its points inside the window, whose sums have one order."""
    import sapa_b200 as sp
    C, d, H, W = shape
    G, P = 4, 9
    t = [_rand(1, B, d, 2 * H, 2 * W, dtype=dtype, scale=0.5), _rand(2, B, d, H, W, dtype=dtype, scale=0.5), _rand(3, B, C, H, W, dtype=dtype),
         _rand(4, B, 2 * G * P, 2 * H, 2 * W, dtype=dtype, scale=0.5).clamp(-1.5, 1.5)]
    go = _rand(5, B, C, 2 * H, 2 * W, dtype=dtype)

    def op(*x):
        return sp.deform_sapa_fused(*x, P, 2, G)
    batch = _results(t, go, op)
    for n in (0, B - 1):
        for i, (a, b) in enumerate(zip(batch, _results([x[n:n + 1] for x in t], go[n:n + 1], op))):
            assert _equal(a[n:n + 1], b, i in (0, 1) and dtype == torch.float32), i      # the output and the query's gradient
