"""Tensor subclasses and torch's modes around a module: what overrides or records torch's ops sees the projections, in training and
inference, and a tensor that keeps its elements elsewhere is never read by its pointer."""
import pytest
import torch
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode
from torch.utils._pytree import tree_map

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class Kept(torch.Tensor):
    """A tensor with no storage of its own, as sharded and quantised parameters are."""

    @staticmethod
    def __new__(cls, inner, requires_grad=False):
        return torch.Tensor._make_wrapper_subclass(cls, inner.shape, dtype=inner.dtype, device=inner.device, requires_grad=requires_grad)

    def __init__(self, inner, requires_grad=False):
        self.inner = inner

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        out = func(*tree_map(lambda a: a.inner if isinstance(a, Kept) else a, args), **tree_map(lambda a: a.inner if isinstance(a, Kept) else a, kwargs or {}))
        return Kept(out) if func is torch.ops.aten.detach.default else out


class Doubled(torch.Tensor):
    """A weight that counts twice in a convolution."""

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        args = [a.as_subclass(torch.Tensor) if isinstance(a, Doubled) else a for a in args]
        if func is torch.conv2d or getattr(func, "__name__", "") == "conv2d":
            args[1] = 2 * args[1]
        return func(*args, **(kwargs or {}))


def _module(cls):
    import sapa_b200
    torch.manual_seed(3)
    m = getattr(sapa_b200, cls)(32, embedding_dim=8 if cls == "SAPA" else 4).to(DEV)
    return m, torch.randn(2, 32, 16, 16, device=DEV), torch.randn(2, 32, 8, 8, device=DEV)


@pytest.mark.parametrize("train", [True, False])
@pytest.mark.parametrize("cls", ["SAPA", "SAPADeform"])
def test_modes_see_the_projections(cls, train):
    m, y, x = _module(cls)

    class Dispatched(TorchDispatchMode):
        seen = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen += func is torch.ops.aten.convolution.default
            return func(*args, **(kwargs or {}))

    class Called(TorchFunctionMode):
        seen = 0

        def __torch_function__(self, func, types, args=(), kwargs=None):
            self.seen += getattr(func, "__name__", "") == "conv2d"
            return func(*args, **(kwargs or {}))
    with torch.set_grad_enabled(train):
        for mode in (Dispatched(), Called()):
            with mode:
                m(y, x)
            assert mode.seen == (2 if cls == "SAPA" else 3)


@pytest.mark.parametrize("train", [True, False])
@pytest.mark.parametrize("cls", ["SAPA", "SAPADeform"])
def test_subclass_parameters(cls, train):
    for subclass in (Kept, Doubled):
        m, y, x = _module(cls)
        plain = m.q.weight.detach()
        with torch.set_grad_enabled(train):
            m.q.weight = torch.nn.Parameter(2 * plain if subclass is Doubled else plain, requires_grad=False)
            want = m(y, x)
            del m.q.weight
            m.q.weight = Kept(plain) if subclass is Kept else plain.as_subclass(Doubled)
            got = m(y, x)
        # float32, the convolutions with TF32 (1e-3) on one side
        assert float((got - want).norm() / want.norm()) < 2e-3


def test_default_device_is_no_reason_to_leave():
    from sapa_b200 import _lib
    m, y, x = _module("SAPA")
    with torch.device(DEV):
        out = m(y, x)
        torch.autograd.grad(out.sum(), list(m.parameters()))
    assert "proj_moments_kernel" in _lib.last_kernels()
