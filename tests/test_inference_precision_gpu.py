"""Inference projections that no q / k kernel served before them - offsets, more than 256 rows - against 64 bits: no further off than
torch's GroupNorm and convolution of the same type, whatever the mean of the features."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _error(t, want):
    return float((t.double() - want).norm() / want.norm())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("mean", [0.0, 3.0, 30.0])
@pytest.mark.parametrize("B,C,HW,d", [(2, 64, 16, 288), (1, 256, 32, 320), (2, 64, 13, 288)])
def test_many_rows_behind_a_norm(B, C, HW, d, mean, dtype):
    from sapa_b200 import _lib
    g = torch.Generator().manual_seed(3)
    x = (torch.randn(B, C, HW, HW, generator=g) + mean).to(dtype).to(DEV)
    w, b = ((torch.randn(*s, generator=g) * f).to(dtype).to(DEV) for s, f in (((d, C, 1, 1), 0.02), ((d,), 0.1)))
    gamma, beta = ((torch.randn(C, generator=g) * 0.1 + s).to(dtype).to(DEV) for s in (1.0, 0.0))

    def ref(t):
        return F.conv2d(F.group_norm(x.to(t), 32, gamma.to(t), beta.to(t), 1e-5), w.to(t), b.to(t))
    want = ref(torch.float64)
    got = _lib.load_host().project_module(x, gamma, beta, 32, 1e-5, w, b, None)
    assert _error(got, want) <= _error(ref(dtype), want)
    # the normalised input, the product and the biased sum are rounded: sqrt(3) half-ulp roundings of mean square 1/12 ulp^2 each, at most
    assert _error(got, want) < 1.2 * torch.finfo(dtype).eps


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("high", [True, False])
def test_offsets_behind_a_norm(high, dtype):
    """The offsets by themselves: their weights grown until they decide the output, features with a mean of 30 deviations."""
    import copy
    import sapa_b200
    torch.manual_seed(2)
    m = sapa_b200.SAPADeform(64, embedding_dim=8, norm=True, high_offset=high)
    with torch.no_grad():
        m.offset.weight.mul_(5)
        m.q.weight.zero_()
    m = m.to(DEV).to(dtype)
    y, x = ((torch.randn(2, 64, s, s, device=DEV) + 30).to(dtype) for s in (32, 16))
    x = x + 4 * torch.randn(2, 64, 1, 1, device=DEV).to(dtype)
    ref, own = copy.deepcopy(m).double(), copy.deepcopy(m)
    ref.impl, own.fuse_projection = "separate", False
    ref.fuse_projection = False
    with torch.no_grad():
        want, got, torchs = ref(y.double(), x.double()), m(y, x), own(y, x)
    mean = x.double().mean((2, 3), keepdim=True)
    assert _error(got.double() - mean, want - mean) <= 1.05 * _error(torchs.double() - mean, want - mean)


@pytest.mark.parametrize("norm", [True, False])
def test_float32_without_tf32_is_torchs(norm, monkeypatch):
    """A caller who has switched TF32 off: 384 rows of q and k, and the offsets, are torch's convolutions, bit for bit."""
    import sapa_b200
    monkeypatch.setattr(torch.backends.cudnn, "allow_tf32", False)
    torch.manual_seed(2)
    m = sapa_b200.SAPADeform(64, embedding_dim=96, norm=norm).to(DEV)
    y, x = (torch.randn(2, 64, s, s, device=DEV) for s in (32, 16))
    with torch.no_grad():
        got = m(y, x)
        m.fuse_projection = False
        assert torch.equal(got, m(y, x))
