"""Kernels of a chain are set up while the previous one drains: calls one after the other, on buffers that the allocator hands on
from call to call, give what each call gives by itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(seed, dtype, W, deform):
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device="cuda") * scale).to(dtype)
    B, C, d, H = 2, 64, 32, 12
    x = [t(B, d, 2 * H, 2 * W, scale=0.5), t(B, d, H, W, scale=0.5), t(B, C, H, W)]
    if deform:
        x.append(t(B, 72, 2 * H, 2 * W, scale=0.3).clamp(-0.9, 0.9))        # no point leaves the window: no atomics
    return [v.requires_grad_() for v in x], t(B, C, 2 * H, 2 * W)


@pytest.mark.parametrize("deform", [False, True], ids=["sapa", "deform"])
@pytest.mark.parametrize("dtype,W", [(torch.float32, 16), (torch.bfloat16, 16), (torch.bfloat16, 17), (torch.float32, 15)])
def test_calls_back_to_back(deform, dtype, W):
    import sapa_b200
    op = (lambda x: sapa_b200.deform_sapa_fused(*x, 9, 2, 4)) if deform else (lambda x: sapa_b200.sapa_fused(*x, 5, 2))

    def one(x, go):
        out = op(x)
        return [out.detach()] + list(torch.autograd.grad(out, x, go))

    cases = [_inputs(s, dtype, W, deform) for s in range(3)]
    alone = []
    for x, go in cases:
        torch.cuda.synchronize()
        alone.append([t.clone() for t in one(x, go)])
        torch.cuda.synchronize()
    # compared on the device and freed, so that the next call gets the memory and nothing waits in between
    atomics = deform and dtype != torch.float32 and W % 8      # the gather/scatter kernels: float32 sums in any order, rounded to 16 bits
    worst = torch.zeros((), device="cuda", dtype=torch.float64)
    for _ in range(5):
        for (x, go), want in zip(cases, alone):
            for u, v in zip(want, one(x, go)):
                worst = torch.maximum(worst, ((u.double() - v.double()).norm() / u.double().norm()) if atomics else (u != v).sum().double())
    assert float(worst) <= (2.0 ** -8 if atomics else 0.0)
