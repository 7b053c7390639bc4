"""Ops and modules under torch.autocast: an op means the same as outside, whichever kernels serve it, and a backward pass inside the
context gives the gradients of one behind it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(*shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(sum(shape))) * scale).to(dtype).to(DEV)


def _call(op, tensors, dtype, on):
    t = [x.clone().requires_grad_() for x in tensors]
    with torch.autocast("cuda", dtype=dtype, enabled=on):
        with torch.no_grad():
            plain = op(*t)
        out = op(*t)
        grads = torch.autograd.grad(out, t, torch.ones_like(out))
    return [plain, out.detach(), *grads]


# the softmax between two separate kernels (no fused kernel for the window, more than 16 points), and the fused kernels
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("K,s", [(7, 2), (5, 4), (3, 3), (5, 2)])
def test_fused_op(K, s, dtype):
    import sapa_b200 as sp
    t = [_rand(1, 8, 6 * s, 6 * s, scale=0.5, dtype=dtype), _rand(1, 8, 6, 6, scale=0.5, dtype=dtype), _rand(1, 12, 6, 6, dtype=dtype)]
    for got, want in zip(*(_call(lambda q, k, v: sp.sapa_fused(q, k, v, K, s), t, dtype, on) for on in (True, False))):
        assert got.dtype == dtype and torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("P", [17, 9])
def test_deform_op(P, dtype):
    import sapa_b200 as sp
    t = [_rand(1, 8, 12, 16, scale=0.5, dtype=dtype), _rand(1, 8, 6, 8, scale=0.5, dtype=dtype), _rand(1, 8, 6, 8, dtype=dtype),
         _rand(1, 4 * P, 12, 16, scale=0.25, dtype=dtype)]
    res = [_call(lambda *a: sp.deform_sapa_fused(*a, P, 2, 2), t, dtype, on) for on in (True, False)]
    for got, want in zip(*res):      # scattered gradients are sums of atomics: float32 sums in another order, then one rounding
        assert got.dtype == dtype and float((got - want).float().norm()) <= 2 * torch.finfo(dtype).eps * float(want.float().norm())


@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("kw", [dict(up_factor=4), dict(up_kernel_size=7)])
def test_module_without_a_fused_kernel(kw, train):
    import sapa_b200
    torch.manual_seed(0)
    m = sapa_b200.SAPA(32, embedding_dim=8, **kw).to(DEV)
    s = kw.get("up_factor", 2)
    y, x = _rand(1, 32, 8 * s, 8 * s), _rand(1, 32, 8, 8)
    with torch.set_grad_enabled(train):
        want = m(y, x)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            got = m(y, x)
    # bfloat16 (4e-3) operands, attention map and output
    assert got.dtype == torch.bfloat16 and float((got - want).norm() / want.norm()) < 2e-2


@pytest.mark.parametrize("cls,kw", [("SAPADeform", dict(high_offset=False)), ("SAPADeform", {}), ("SAPA", {}), ("SAPADeform", dict(num_point=17))])
def test_backward_inside_the_context(cls, kw):
    import sapa_b200
    torch.manual_seed(0)
    m = getattr(sapa_b200, cls)(32, embedding_dim=8, **kw).to(DEV)
    t = [_rand(1, 32, 16, 16).requires_grad_(), _rand(1, 32, 8, 8).requires_grad_(), *m.parameters()]
    grads = []
    for inside in (False, True):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = m(t[0], t[1])
            if inside:
                grads.append(torch.autograd.grad(out, t, torch.ones_like(out)))
        if not inside:
            grads.append(torch.autograd.grad(out, t, torch.ones_like(out)))
    scale = max(float(g.norm()) for g in grads[0])      # atomics, as above, rounded to bfloat16 (4e-3) on the way; a key bias cancels
    for got, want in zip(grads[1], grads[0]):
        assert float((got - want).norm()) <= 1e-2 * float(want.norm()) + 1e-3 * scale
