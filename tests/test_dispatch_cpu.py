"""Which calls the CUDA wrappers hand to a kernel and which they leave to the general path, without
a GPU: the kernel library is a stand-in that notes its calls."""
from types import SimpleNamespace

import pytest
import torch

from rvllm_b200.errors import KernelError
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


@pytest.fixture
def split_ops(ops):
    ops.split = []
    ops.lib.rv_gemm_f32_better = lambda M, N, K: 0
    ops.lib.rv_gemm_f32_split_scratch = lambda m, k: 8
    ops.lib.rv_gemm_f32_split = lambda *a: ops.split.append(a) or 0
    ops._gemm_status = lambda device: torch.zeros(1, dtype=torch.int32)
    return ops


@pytest.mark.parametrize("m,n,k,taken", [
    (1, 256, 512, True), (32, 256, 768, True), (33, 256, 768, True), (33, 1024, 768, True), (2048, 1024, 768, True),
    (8, 255, 768, False), (8, 2048, 508, False), (8, 2048, 764, True), (8, 2048, 770, False)])
def test_float32_product_of_parts_by_size(split_ops, m, n, k, taken):
    split_ops.linear(on_device(m, k), on_device(n, k))
    assert len(split_ops.split) == int(taken) and not split_ops.calls
    split_ops.lib.rv_gemm_f32_better = lambda M, N, K: 1    # the other kernel is asked first
    split_ops.linear(on_device(m, k), on_device(n, k))
    assert len(split_ops.split) == int(taken) and len(split_ops.calls) == 1


def test_float32_product_of_parts_leaves_more_columns_than_a_grid_has():
    assert CudaOps._split_better(8, 65535 * 128, 1024) and not CudaOps._split_better(8, 65535 * 128 + 1, 1024)


def test_float32_product_of_parts_takes_what_fits(split_ops):
    """Operands with other strides, of other types, at other addresses, on other devices or that want
    gradients stay with the library; what it refuses stays refused."""
    x, w = on_device(8, 1024), on_device(512, 1024)
    for a, b in ((on_device(1024, 8).t(), w), (x, on_device(1024, 512).t()), (on_device(8, 2048)[:, ::2], w),
                 (on_device(8 * 1024 + 1)[1:].view(8, 1024), w), (x, on_device(512, 1024, number=1)),
                 (x, on_device(512, 1024, grad=True)), (x.double(), w.double())):
        y = split_ops.linear(a, b)
        assert not split_ops.split and not split_ops.calls
        assert torch.allclose(torch.Tensor(y.detach().float()), torch.Tensor((a @ b.t()).detach().float()), atol=1e-3)
    for a, b in ((x, on_device(512, 2048)), (on_device(2, 8, 1024), w), (x, on_device(2, 512, 1024))):
        with pytest.raises((RuntimeError, ValueError)):
            split_ops.linear(a, b)
    assert not split_ops.split
    split_ops.linear(x, w)
    split_ops.linear(x, w.bfloat16())                       # cast, then multiplied
    assert len(split_ops.split) == 2


@pytest.mark.parametrize("code", [12, 33, 45])
def test_a_wait_that_ran_out_is_named_wherever_it_is_asked_for(ops, code):
    word = torch.tensor([code], dtype=torch.int32)
    ops._gemm_state = {"cuda:0": word}
    with pytest.raises(KernelError, match=f"code {code}:.*31-34 grouped experts, 41-45 float32 products.* on cuda:0"):
        ops.check_status()
    assert int(word) == 0
    with pytest.raises(KernelError, match=f"code {code}:.*31-34 grouped experts, 41-45 float32 products"):
        ops.raise_for_status(code)
    ops.check_status()
    ops.raise_for_status(0)


class Cuda(OnDevice):
    is_cuda = True


def cuda(*shape, dtype=torch.float32):
    return torch.zeros(*shape, dtype=dtype).as_subclass(Cuda)


def forms(ops, lens, longest=None, heads=8, dim=64, singles=0, reqs=None):
    """Whether a step of these portions takes the chunk forms of the matrix memory and of the delta
    rule with a decay per channel; `longest`, `reqs`: what the step says, when it is padded."""
    n, taken = sum(lens) + singles, {}
    ctx = SimpleNamespace(n_decode=singles, n_reqs=singles + (reqs or len(lens)), max_q_len=longest or max(lens),
                          token_req=None, q_start=None, state_slot=None)
    value = lambda a: a.value if hasattr(a, "value") else a
    ops.mlstm_mode, ops.mlstm_above, ops.gated_delta_mode, ops.gated_delta_above = "auto", 384, "chunks", 288
    ops.lib.rv_mlstm_chunks_ok = lambda *a: 1
    ops.lib.rv_mlstm_scratch = ops.lib.rv_gated_delta_scratch = lambda *a: 0
    ops.lib.rv_mlstm = lambda *a: taken.update(memory=bool(value(a[-2]))) or 0
    ops.lib.rv_gated_delta = lambda *a: taken.update(delta=bool(value(a[-2]))) or 0
    ops.mlstm(cuda(n, 4 * heads * dim + 2 * heads), cuda(heads), cuda(heads), cuda(heads * dim),
              cuda(1, heads * (dim + 1) * dim + heads), ctx, cuda(n, heads * dim, dtype=torch.bfloat16),
              heads, dim, dim, 5.0, 1e-5)
    C = 3 * heads * dim
    ops.gated_delta(cuda(n, C + heads), cuda(n, 2 * heads * dim), cuda(C, 4), cuda(heads), cuda(heads * dim),
                    cuda(dim), cuda(1, 3 * C + heads * dim * dim), ctx, cuda(n, heads * dim, dtype=torch.bfloat16),
                    heads, heads, dim, dim, 4, 1e-6, 1e-5)
    return taken["memory"], taken["delta"]


def test_chunk_forms_are_for_long_portions(ops):
    """By the longest portion, not by the tokens of all; the delta rule's also by how full its chunks
    are and, for small heads, by whether the scan waits for the longest portion alone."""
    assert forms(ops, [60] * 8) == (False, False)
    assert forms(ops, [288]) == (False, False) and forms(ops, [384]) == (False, True)
    assert forms(ops, [400]) == (True, True) and forms(ops, [1489, 559]) == (True, True)
    assert forms(ops, [400] + [16] * 31) == (True, False)
    assert forms(ops, [400], singles=31) == (True, True)
    assert forms(ops, [400] * 8) == (True, False)
    assert forms(ops, [400] * 8, dim=128) == (True, True)
    assert forms(ops, [400] * 8, dim=128, heads=16) == (True, True)


def sizes_of(lens, limits, shallow=0, context=0, page=16):
    from rvllm_b200.engine.batch import StepEntry
    from rvllm_b200.engine.runner import ModelRunner
    r = object.__new__(ModelRunner)
    r._portion_limits, r._shallow = limits, shallow
    r.cache = SimpleNamespace(page_size=page, requests={i: SimpleNamespace(computed=context) for i in range(len(lens))})
    return r._mixture_sizes([StepEntry(i, (0,) * n, (0,)) for i, n in enumerate(lens)])


@pytest.mark.parametrize("lens", [[60] * 8, [40] * 8, [1] * 8 + [48] * 10, [288], [289], [300, 20, 20], [384], [385],
                                  [400], [700], [2000], [1, 1, 1, 260], [257, 257, 257], [30] * 31])
def test_padded_steps_choose_as_exact_ones(ops, lens):
    """What a padded step tells the kernels about its longest portion chooses the same form of the
    matrix memory as the portions themselves, and covers every request's tokens, the filling ones
    included; the delta rule's may stay with the scan, but takes chunks only where the portions do."""
    single = sum(n == 1 for n in lens)
    portions = lens[single:]
    D, P, T, _, longest, deepest = sizes_of(lens, (288, 384))
    assert longest >= max(portions) and longest >= T - D - sum(portions) and longest <= T - D
    assert deepest == sizes_of(lens, None)[5] and sizes_of(lens, None)[4] == T - D
    tail = [T - D - sum(portions)]
    for dim in (64, 128):
        exact = forms(ops, portions, singles=single, dim=dim)
        padded = forms(ops, portions + tail, longest=longest, singles=D, reqs=P, dim=dim)
        assert padded[0] == exact[0] and padded[1] <= exact[1], (dim, exact, padded)


def test_padded_steps_of_shallow_contexts():
    """Where attention has another kernel for short contexts, steps within them are told so."""
    assert sizes_of([20, 30], (), shallow=64)[5] == 64
    assert sizes_of([20, 30], (), shallow=64, context=34)[5] == 64
    assert sizes_of([20, 30], (), shallow=64, context=35)[5] == 256
    assert sizes_of([20, 30], None, shallow=0)[5] == 256
    assert sizes_of([20, 30], (), shallow=64, page=2)[5] == 32


@pytest.mark.parametrize("lens,context,window,better", [
    ([300], 300, None, True), ([20, 30], 30, None, False), ([500] + [20] * 15, 500, None, True),
    ([500] + [20] * 31, 500, None, False), ([1000] + [20] * 63, 1000, None, False), ([70] + [10] * 31, 70, None, False),
    ([66] * 31, 66, None, True), ([4] * 31, 504, None, True), ([500] + [20] * 31, 800, None, True),
    ([500] + [20] * 31, 800, 10, False), ([2] * 8192, 5000, None, False),
    ([70000], 70000, None, False)])
def test_prefill_kernel_for_heads_of_128(ops, lens, context, window, better):
    """By how much of what is launched has tokens, and by the depth of the context; more portions,
    or longer ones, than the tcgen05 kernel's grid has are left to the other kernel, which takes them."""
    ctx = SimpleNamespace(n_reqs=len(lens) + 3, n_tokens=sum(lens) + 3, max_q_len=max(lens), max_ctx_len=context)
    assert ops._tcgen05_better_128(ctx, 3, window) is better
