"""Chains of kernels that are set up while the previous one drains: modules and deformable ops, back to back on memory that goes from call to
call, against float64 and against the same calls with the GPU idle before each."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = {torch.float32: 1e-5, torch.bfloat16: 2e-2, torch.float16: 4e-3}      # 2-norm against float64: see test_outlier_lists_gpu.py


def _rand(g, *shape, scale=1.0):
    return torch.randn(*shape, generator=g, device=DEV) * scale


def _apart(a, b):
    """Relative difference in the 2-norm, on the device: no wait between the calls that are compared."""
    return (a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)


def _back_to_back(calls, alone, tol, rounds=4):
    """Each call several times in turn; its results are compared on the device and freed, so that the next call gets their memory."""
    worst = [torch.zeros((), device=DEV, dtype=torch.float64)]
    for _ in range(rounds):
        for call, want in zip(calls, alone):
            for a, b in zip(call(), want):
                worst.append(torch.maximum(worst.pop(), _apart(a, b) if tol else (a != b).sum().double()))
    assert float(worst[0]) <= tol


def _alone(call):
    torch.cuda.synchronize()
    out = [t.clone() for t in call()]
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("separate", [False, True])
def test_lists_of_far_points_long_and_empty_in_turn(separate, dtype):
    """A counter or a list that is read too early shows: the lists are long, empty, short in turn."""
    import sapa_b200 as sp
    B, C, d, H, W, G, P = 2, 32, 16, 24, 32, 4, 9
    calls, doubles = [], []
    sigmas = (1.5, 0.2, 0.7, 0.1)
    for n, sigma in enumerate(sigmas):
        g = torch.Generator(device=DEV).manual_seed(n)
        o = (_rand(g, B, 2 * P * G, 2 * H, 2 * W, scale=sigma) * 64).round() / 64 + 1 / 128      # positions are exact in float32
        t = [x.to(dtype) for x in (_rand(g, B, d, 2 * H, 2 * W, scale=0.5), _rand(g, B, d, H, W, scale=0.5), _rand(g, B, C, H, W), o)]
        a, ga, go = (x.to(dtype) for x in (torch.rand(B, G, P, 2 * H, 2 * W, generator=g, device=DEV), _rand(g, B, G, P, 2 * H, 2 * W), _rand(g, B, C, 2 * H, 2 * W)))

        def call(t=t, a=a, ga=ga, go=go, double=False):
            q, k, v, o, a, ga, go = (x.double() if double else x for x in (*t, a, ga, go))
            q, k, v, o, a = (x.detach().requires_grad_() for x in (q, k, v, o, a))
            if separate:
                sim, out = sp.deform_qk(q, k, o, P, 2, G), sp.deform_av(a, v, o, P, 2, G)
                return [sim.detach(), out.detach(), *torch.autograd.grad(sim, (q, k, o), ga), *torch.autograd.grad(out, (a, v, o), go)]
            out = sp.deform_sapa_fused(q, k, v, o, P, 2, G)
            return [out.detach(), *torch.autograd.grad(out, (q, k, v, o), go)]
        calls.append(call)
        doubles.append(call(double=True))
    alone = [_alone(c) for c in calls]
    # dS = A (dA - sum A dA): the rounding of A leaves the sum an ulp off, against differences of dA that shrink with the offsets' spread
    for got, want, sigma in zip(alone, doubles, sigmas):
        errors = [float(_apart(a, b)) for a, b in zip(got, want)]
        assert max(errors) < TOL[dtype] * max(1.0, 0.2 / sigma), (sigma, errors)
    # the far points' gradients are added by atomics, in any order: the bound is the one against float64; what has no atomics is the same bit by bit
    _back_to_back(calls, alone, TOL[dtype])
    forward = (lambda c: (lambda: c()[:2])) if separate else (lambda c: (lambda: c()[:1]))
    _back_to_back([forward(c) for c in calls], alone, 0)
    _back_to_back([calls[3]], [alone[3]], 0)


@pytest.mark.parametrize("kind", ["SAPA", "SAPADeform"])
@pytest.mark.parametrize("mode", ["f32", "f16", "bf16", "train_f32", "train_amp"])
def test_modules(kind, mode):
    import sapa_b200 as sp
    train, amp = mode.startswith("train"), mode.endswith("amp")
    dtype = {"f16": torch.float16, "bf16": torch.bfloat16}.get(mode, torch.float32)
    torch.manual_seed(5)
    module = (sp.SAPA(64, 64, embedding_dim=32) if kind == "SAPA" else sp.SAPADeform(64, 64, embedding_dim=32, norm=True)).to(DEV, dtype)
    reference = (sp.SAPA(64, 64, embedding_dim=32) if kind == "SAPA" else sp.SAPADeform(64, 64, embedding_dim=32, norm=True)).to(DEV).double()
    reference.load_state_dict({k: v.double() for k, v in module.state_dict().items()})
    calls, doubles = [], []
    for n, H in enumerate((16, 8, 24)):
        g = torch.Generator(device=DEV).manual_seed(n)
        y, x, go = (t.to(dtype) for t in (_rand(g, 2, 64, 2 * H, 32), _rand(g, 2, 64, H, 16), _rand(g, 2, 64, 2 * H, 32)))

        def call(m=module, y=y, x=x, go=go, double=False):
            if double:
                m, y, x, go = reference, y.double(), x.double(), go.double()
            if not train:
                with torch.no_grad():
                    return [m(y, x)]
            y, x = y.detach().requires_grad_(), x.detach().requires_grad_()
            with torch.autocast("cuda", torch.bfloat16, enabled=amp and not double):
                out = m(y, x)
            return [out.detach(), *torch.autograd.grad(out, [y, x, *m.parameters()], go.to(out.dtype))]
        calls.append(call)
        doubles.append(call(double=True))
    alone = [_alone(c) for c in calls]
    # float32: the products' 7e-6 behind a norm, times logits (or offsets) of a few units in the exponent and in the weights: 1e-4; 16
    # bits: every step of the sequence rounds.  The output alone: gradients behind a rounded query have no such bound
    for got, want in zip(alone, doubles):
        assert float(_apart(got[0], want[0])) < (4e-2 if amp or dtype == torch.bfloat16 else 1e-2 if dtype == torch.float16 else 1e-4)
    _back_to_back(calls, alone, 0 if kind == "SAPA" or not train else 2e-2 if amp else 1e-4)


def test_captured_chain_with_far_points():
    """The same launches as nodes of a CUDA graph: replayed with lists of other lengths."""
    import sapa_b200 as sp
    B, C, d, H, W, G, P = 2, 32, 16, 24, 32, 4, 9

    def inputs(sigma):
        g = torch.Generator(device=DEV).manual_seed(3)
        return [_rand(g, B, d, 2 * H, 2 * W, scale=0.5), _rand(g, B, d, H, W, scale=0.5), _rand(g, B, C, H, W), _rand(g, B, 2 * P * G, 2 * H, 2 * W, scale=sigma)]
    with torch.no_grad():
        graphed = sp.GraphedForward(lambda q, k, v, o: sp.deform_sapa_fused(q, k, v, o, P, 2, G), inputs(0.2))
        for sigma in (1.5, 0.2, 1.5, 0.0):
            t = inputs(sigma)
            assert torch.equal(graphed(*t), sp.deform_sapa_fused(*t, P, 2, G))
