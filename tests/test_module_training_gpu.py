"""Training through the native module path (projections and attention in one autograd node): outputs and every gradient against
the same module in float64 on the separate ops, at the sizes where the projection kernels' tiles, slices and rows end."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# class, B, C, embedding_dim, H, W, constructor arguments: rows of 16 bytes and others, channel and pixel tails, one group per
# channel, more than one slice of pixels, no bias, no norm, more than 256 offset rows, low-resolution offsets
CASES = [("SAPA", 2, 64, 16, 8, 8, {}), ("SAPA", 2, 96, 48, 7, 9, {}), ("SAPA", 3, 32, 32, 5, 6, dict(qkv_bias=False)),
         ("SAPA", 1, 128, 32, 48, 40, {}), ("SAPA", 2, 72, 24, 4, 5, dict(norm=False)), ("SAPADeform", 2, 64, 16, 8, 8, {}),
         ("SAPADeform", 1, 32, 8, 7, 5, dict(norm=True)), ("SAPADeform", 2, 32, 8, 6, 4, dict(high_offset=False))]


def _run(m, y, x, go, amp):
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=amp):
        out = m(y, x)
    return [out.detach()] + list(torch.autograd.grad(out, [y, x] + list(m.parameters()), go.to(out.dtype)))


@pytest.mark.parametrize("mode", ["float32", "amp"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "%s_B%d_C%d_e%d_%dx%d_%s" % (*c[:6], "_".join(c[6])))
def test_module_gradients(case, mode, monkeypatch):
    import sapa_b200
    from sapa_b200 import _lib
    cls, B, C, e, H, W, kw = case
    # float32 offsets are torch's convolution: compared without tf32, where the whole module is left to torch's projections
    native = mode == "amp" or cls == "SAPA"
    monkeypatch.setattr(torch.backends.cudnn, "allow_tf32", native)
    g = torch.Generator().manual_seed(7)
    m = getattr(sapa_b200, cls)(C, embedding_dim=e, **kw)
    with torch.no_grad():
        for name, p in m.named_parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.05 if p.dim() > 1 else 0.2) + (1 if "norm" in name and "weight" in name else 0))
    m = m.to(DEV)
    y, x = (torch.randn(B, C, *s, generator=g).to(DEV).requires_grad_() for s in ((2 * H, 2 * W), (H, W)))
    go = torch.randn(B, C, 2 * H, 2 * W, generator=g).to(DEV).bfloat16().float()
    ref = copy.deepcopy(m).double()
    ref.impl, ref.fuse_projection = "separate", False
    want = _run(ref, y.detach().double().requires_grad_(), x.detach().double().requires_grad_(), go.double(), False)
    got = _run(m, y, x, go, mode == "amp")
    assert ("proj_moments_kernel" in _lib.last_kernels()) == native
    names = ["out", "y", "x"] + [n for n, _ in m.named_parameters()]
    for name, a, b in zip(names, got, want):
        rel = float((a.double() - b).norm() / b.norm())
        # float32: a few rounded steps in a chain of three-term tf32 products (1e-6 each), with logits of a few units.  amp:
        # bfloat16 (4e-3) attention operands and gradients; what follows the offsets is differentiated through bilinear
        # corners whose choice an offset rounded to bfloat16 changes, and the key bias / norm gradients cancel over the window
        if mode == "float32":
            tol = 5e-5
        else:
            tol = 0.3 if cls == "SAPADeform" and (name == "x" or "offset" in name or "norm_x" in name) else 0.1 if name in ("k.bias", "norm_x.bias") else 2e-2
        assert rel < tol, (name, rel)
    assert _lib.wait_timeout_flags(DEV) == 0


@pytest.mark.parametrize("mode", ["float32", "amp"])
@pytest.mark.parametrize("kw", [dict(), dict(norm=True), dict(high_offset=False), dict(norm=True, high_offset=False, qkv_bias=False)],
                         ids=lambda k: "_".join(k) or "plain")
@pytest.mark.parametrize("H,W", [(8, 8), (7, 5)])
def test_deform_module_gradients_inside_cells(H, W, kw, mode):
    """Every gradient of the native SAPADeform node, where it can be held to the rounding: offsets that the features move little and the
    bias keeps in the middle of a cell, so that no rounding changes a bilinear corner."""
    import sapa_b200
    g = torch.Generator().manual_seed(7)
    B, C, e, P, G = 2, 64, 8, 3, 2
    m = sapa_b200.SAPADeform(C, embedding_dim=e, num_point=P, groups=G, **{**kw, "qkv_bias": True})
    with torch.no_grad():
        for name, p in m.named_parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (0.05 if p.dim() > 1 else 0.2) + (1 if "norm" in name and "weight" in name else 0))
        m.offset.weight.mul_(0.2)
        # pixels lie on whole cells: the middle of one of the four around each, per point
        m.offset.bias.copy_(torch.randint(0, 2, m.offset.bias.shape, generator=g) - 0.5)
        if not kw.get("qkv_bias", True):
            m.q.bias = m.k.bias = None
    m = m.to(DEV)
    y, x = (torch.randn(B, C, *s, generator=g).to(DEV).requires_grad_() for s in ((2 * H, 2 * W), (H, W)))
    go = torch.randn(B, C, 2 * H, 2 * W, generator=g).to(DEV).bfloat16().float()
    ref = copy.deepcopy(m).double()
    ref.impl, ref.fuse_projection = "separate", False
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=mode == "amp"):
        assert "DeformModuleNode" in m(y, x).grad_fn.name()
    want = _run(ref, y.detach().double().requires_grad_(), x.detach().double().requires_grad_(), go.double(), False)
    got = _run(m, y, x, go, mode == "amp")
    # float32: offsets without a norm are torch's convolution with TF32 (1e-3 of an offset's part that the features make, 0.05),
    # the rest three-term products (1e-6).  amp: bfloat16 (4e-3) operands, offsets rounded to steps of 2^-9 around a half,
    # attention and gradients; norms and key biases cancel in part
    names = ["out", "y", "x"] + [n for n, _ in m.named_parameters()]
    for name, a, b in zip(names, got, want):
        rel = float((a.double() - b).norm() / b.norm())
        tol = (2e-4 if mode == "float32" else 2e-2) * (3 if name in ("k.bias", "norm_x.bias", "norm_x.weight") else 1)
        assert rel < tol, (name, rel)
