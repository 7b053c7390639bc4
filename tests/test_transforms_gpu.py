"""What torch wraps around an op or a module - traces, forward-mode differentiation, torch.func, hooks, overridden methods, a
backward that is differentiated - is seen by the native host path: the same results, or the same refusal, as from autograd
Functions and torch modules."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(grad=False):
    g = torch.Generator().manual_seed(11)
    q, k, v, o = (torch.randn(*s, generator=g).to(DEV) for s in ((1, 8, 8, 16), (1, 8, 4, 8), (1, 8, 4, 8), (1, 36, 8, 16)))
    o = 0.25 * o      # points inside the window: gradients without atomics
    return [t.requires_grad_(grad) for t in (q, k, v, o)]


def _ops():
    import sapa_b200 as sp
    return {"fused": lambda q, k, v, o: sp.sapa_fused(q, k, v, 5, 2),
            "separate": lambda q, k, v, o: sp.av(torch.softmax(sp.qk(q, k, 5, 2), dim=1), v, 5, 2),
            "deform": lambda q, k, v, o: sp.deform_sapa_fused(q, k, v, o, 9, 2, 2),
            "deform_separate": lambda q, k, v, o: sp.deform_av(torch.softmax(sp.deform_qk(q, k, o, 9, 2, 2), dim=2), v, o, 9, 2, 2)}


@pytest.mark.parametrize("name", ["fused", "separate", "deform", "deform_separate"])
def test_ops_under_transforms(name):
    op = _ops()[name]
    t = _inputs(True)
    want = torch.autograd.grad(op(*t).square().sum(), t, allow_unused=True)
    traced = torch.jit.trace(op, tuple(_inputs(True)), check_trace=False)
    other = [x.detach().flip(0, 2).requires_grad_() for x in t]
    assert torch.equal(traced(*other), op(*other))
    got = torch.autograd.grad(traced(*t).square().sum(), t, allow_unused=True)
    for a, b in zip(got, want):
        assert (a is None and b is None) or torch.equal(a, b)
    plain = _inputs()
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda q: op(q, *plain[1:]).sum())(plain[0])
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda q: op(q, *plain[1:]))(plain[0][None])
    with torch.autograd.forward_ad.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
        op(torch.autograd.forward_ad.make_dual(plain[0], plain[0]), *plain[1:])


def _module(cls, **kw):
    import sapa_b200
    torch.manual_seed(3)
    m = getattr(sapa_b200, cls)(32, embedding_dim=8, **kw).to(DEV)
    return m, torch.randn(2, 32, 8, 16, device=DEV), torch.randn(2, 32, 4, 8, device=DEV)


@pytest.mark.parametrize("cls", ["SAPA", "SAPADeform"])
def test_modules_keep_what_is_around_them(cls):
    m, y, x = _module(cls)
    want = m(y, x)
    seen = []
    for what in ("register_forward_hook", "register_full_backward_hook", "register_full_backward_pre_hook"):
        for sub in [m.q, m.k] + ([m.norm_x] if cls == "SAPA" else []):
            handle = getattr(sub, what)(lambda *a: seen.append(what))
            out = m(y.requires_grad_(), x.requires_grad_())
            out.sum().backward()
            handle.remove()
            assert seen and torch.allclose(out, want, rtol=1e-2, atol=1e-2)
            seen.clear()

    class Scaled(type(m)):
        def attention(self, *a):
            return 2 * super().attention(*a)
    s = copy.deepcopy(m)
    s.__class__ = Scaled
    assert torch.allclose(s(y, x), 2 * want, rtol=1e-2, atol=1e-2)
    traced = torch.jit.trace(m, (y, x), check_trace=False)
    assert torch.allclose(traced(y.flip(0), x.flip(0)), want.flip(0), rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("amp", [False, True])
@pytest.mark.parametrize("cls,kw", [("SAPA", {}), ("SAPA", dict(qkv_bias=False)), ("SAPADeform", {}), ("SAPADeform", dict(norm=True)),
                                    ("SAPADeform", dict(high_offset=False))])
def test_module_gradients_stay_differentiable(cls, kw, amp):
    """create_graph through the native nodes: the projections' part of the gradients carries a graph, as with torch's modules around
    the op (whose own gradients are constants there): a gradient penalty gives the same second gradients."""
    m, y, x = _module(cls, **kw)
    if cls == "SAPADeform":       # small embeddings, for 64 rows behind a norm at most; offsets away from the borders between cells
        import sapa_b200
        m = sapa_b200.SAPADeform(32, embedding_dim=4, num_point=3, groups=2, **kw).to(DEV)
        with torch.no_grad():
            m.offset.weight.mul_(0.1)
            m.offset.bias.copy_(torch.rand(m.offset.bias.shape, generator=torch.Generator().manual_seed(5)) * 0.2 + 0.1)
    ref = copy.deepcopy(m)
    ref.fuse_projection = False
    res = []
    for mod in (m, ref):
        a, b = y.clone().requires_grad_(), x.clone().requires_grad_()
        # the float32 reference in float32, where the native path has three-term products
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=amp), torch.backends.cudnn.flags(allow_tf32=mod is m or amp):
            out = mod(a, b)
            if mod is m:
                assert ("SapaModuleNode" if cls == "SAPA" else "DeformModuleNode") in out.grad_fn.name()
            first = torch.autograd.grad(out.float().square().sum(), [a, b] + list(mod.parameters()), create_graph=True)
            second = torch.autograd.grad(sum(f.square().sum() for f in first), [a, b] + list(mod.parameters()), allow_unused=True)
        res.append((first, second))
    # float32: the recorded gradients are torch's convolutions with TF32 on the native side (1e-3, twice in the second gradients).
    # amp: both sides round to bfloat16 (4e-3) at the same places
    for got, want in zip(*res):
        scale = max(float(s.detach().norm()) for s in want if s is not None)
        for f, w in zip(got, want):
            assert (f is None) == (w is None)
            if w is not None:
                assert float((f - w).detach().norm()) <= (1e-2 if amp else 4e-3) * float(w.detach().norm()) + 1e-4 * scale


def test_parameters_elsewhere_are_refused():
    """The native path reads parameters by pointer: what is not whole, or not on the input's device, is left to torch's checks."""
    m, y, x = _module("SAPA")
    with torch.no_grad():
        m.q.cpu()
        with pytest.raises(RuntimeError):
            m(y, x)
        from sapa_b200.projection import project
        with pytest.raises((RuntimeError, NotImplementedError)):
            project(y, m.norm_y, m.q)
        m.q.to(DEV)
        m.norm_x = torch.nn.GroupNorm(4, 16).to(DEV)
        with pytest.raises(RuntimeError):
            m(y, x)
