"""Which calls the CUDA wrappers hand to a kernel and which they leave to the general path, without
a GPU: the kernel library is a stand-in that notes its calls."""
from types import SimpleNamespace

import pytest
import torch

from rvllm_b200.kernels.bindings import CudaOps


class OnDevice(torch.Tensor):
    """A tensor in host memory that says it is on a device."""

    def get_device(self):
        return getattr(self, "number", 0)


def on_device(*shape, number=0, grad=False):
    t = torch.randn(*shape).as_subclass(OnDevice)
    t.number = number
    return t.requires_grad_(grad)


@pytest.fixture
def ops(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    o = object.__new__(CudaOps)
    o.calls, o.launches = [], 0
    o.gemm_mode, o.gemm_small_m, o.gemm_row_pad = "tcgen05", 16, 1
    o._stream = lambda: None
    o.lib = SimpleNamespace(rv_gemm_f32_better=lambda M, N, K: 1,
                            rv_gemm_f32=lambda *a: o.calls.append(a) or 0)
    return o


def test_float32_product_takes_what_fits(ops):
    ops.linear(on_device(8, 512), on_device(300, 512))
    assert len(ops.calls) == 1


@pytest.mark.parametrize("x,w", [((8, 512), (300, 256)), ((8, 512), (300, 1024)), ((2, 512, 512), (300, 512)),
                                 ((8, 512), (2, 300, 512))])
def test_float32_product_refuses_what_does_not_fit(ops, x, w):
    """Rows and a matrix of other inner sizes, or with more dimensions, are refused as the library
    refuses them; the kernel, which would read beyond the shorter one, is not called."""
    with pytest.raises((RuntimeError, ValueError)):
        ops.linear(on_device(*x), on_device(*w))
    assert not ops.calls


def test_float32_product_leaves_other_devices_and_gradients(ops):
    """Operands of another device than the current one, and such as want gradients, go to the
    library."""
    for x, w in ((on_device(8, 512, number=1), on_device(300, 512, number=1)),
                 (on_device(8, 512), on_device(300, 512, number=1)),
                 (torch.randn(8, 512), torch.randn(300, 512)),
                 (on_device(8, 512), on_device(300, 512, grad=True))):
        y = ops.linear(x, w)
        assert not ops.calls and y.shape == (8, 300)
    assert y.requires_grad
    with torch.no_grad():
        ops.linear(on_device(8, 512), on_device(300, 512, grad=True))
    assert len(ops.calls) == 1
