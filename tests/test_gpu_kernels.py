"""Each CUDA kernel alone against its plain reference (tests/plain_ops.py), at sizes
other than the engine's: widths that are no power of two, head sizes 48 and 80, groups
of 3, pages of 8, filters of 2 to 5 taps."""
import math
import os
import random
import subprocess
import sys
from ctypes import c_int
from types import SimpleNamespace

import pytest
import torch

from plain_ops import PlainOps, sample_row, uniform
from rvllm_b200.kernels.bindings import _ptr

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]


@pytest.fixture(scope="module")
def ops():
    from rvllm_b200.kernels import cuda_ops
    return cuda_ops()


def tol(dtype):
    return dict(atol=2e-6, rtol=2e-6) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)


def rnd(shape, dtype, gen, scale=1.0):
    return (torch.randn(shape, generator=gen) * scale).to(dtype)


@pytest.mark.parametrize("dtype", DTYPES)
def test_embed(ops, dtype):
    g = torch.Generator().manual_seed(1)
    table = rnd((777, 200), dtype, g)
    ids = torch.randint(0, 777, (37,), generator=g, dtype=torch.int32)
    ref = torch.empty(37, 200)
    PlainOps().embed(table, ids, ref, 1.5)
    out = torch.empty(37, 200, device="cuda")
    ops.embed(table.cuda(), ids.cuda(), out, 1.5)
    assert torch.equal(out.cpu(), ref)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("hidden", [200, 1000, 2048])
def test_add_rmsnorm(ops, dtype, hidden):
    g = torch.Generator().manual_seed(2)
    resid = rnd((19, hidden), torch.float32, g)
    delta = rnd((19, hidden), dtype, g)
    w = 1 + rnd((hidden,), torch.float32, g, 0.05)
    for use_delta in (True, False):
        r_ref, out_ref = resid.clone(), torch.empty(19, hidden, dtype=dtype)
        PlainOps().add_rmsnorm(r_ref, delta if use_delta else None, w, 1e-5, out_ref)
        r_gpu, out = resid.cuda(), torch.empty(19, hidden, dtype=dtype, device="cuda")
        ops.add_rmsnorm(r_gpu, delta.cuda() if use_delta else None, w.cuda(), 1e-5, out)
        assert torch.allclose(r_gpu.cpu(), r_ref, atol=1e-6, rtol=1e-6)
        assert torch.allclose(out.cpu().float(), out_ref.float(), **tol(dtype))
    rows = torch.tensor([3, 18, 0, 3], dtype=torch.int32)
    out_ref = torch.empty(4, hidden, dtype=dtype)
    PlainOps().add_rmsnorm(resid.clone(), delta, w, 1e-6, out_ref, rows)
    r_gpu, out = resid.cuda(), torch.empty(4, hidden, dtype=dtype, device="cuda")
    ops.add_rmsnorm(r_gpu, delta.cuda(), w.cuda(), 1e-6, out, rows.cuda())
    assert torch.equal(r_gpu.cpu(), resid)          # stream untouched with a row list
    assert torch.allclose(out.cpu().float(), out_ref.float(), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("ffn", [200, 1024])
def test_swiglu(ops, dtype, ffn):
    g = torch.Generator().manual_seed(3)
    x = rnd((13, 2 * ffn), dtype, g, 2.0)
    ref = torch.empty(13, ffn, dtype=dtype)
    PlainOps().swiglu(x, ref)
    out = torch.empty(13, ffn, dtype=dtype, device="cuda")
    ops.swiglu(x.cuda(), out)
    assert torch.allclose(out.cpu().float(), ref.float(), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
def test_add_bias(ops, dtype):
    g = torch.Generator().manual_seed(4)
    x, b = rnd((11, 77), dtype, g), rnd((77,), torch.float32, g)
    ref = x.clone()
    PlainOps().add_bias(ref, b)
    out = x.cuda()
    ops.add_bias(out, b.cuda())
    assert torch.allclose(out.cpu().float(), ref.float(), **tol(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
def test_linear_float32_is_float32(ops, dtype):
    g = torch.Generator().manual_seed(5)
    x, w = rnd((33, 300), dtype, g), rnd((70, 300), dtype, g)
    ref = x.double() @ w.double().t()
    out = ops.linear(x.cuda(), w.cuda(), out_dtype=torch.float32).cpu().double()
    # float32 operands: errors of float32 accumulation only (TF32 would give ~1e-3)
    bound = 2e-5 if dtype == torch.float32 else 2e-5
    assert (out - ref).abs().max() <= bound * ref.abs().max()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("norm,rope", [(True, True), (False, True), (True, False)])
def test_qk_norm_rope_write(ops, dtype, norm, rope):
    g = torch.Generator().manual_seed(6)
    nh, nkv, hd, n, ps, pages = 6, 2, 48, 21, 8, 9
    qkv = rnd((n, (nh + 2 * nkv) * hd), dtype, g)
    qw = (1 + rnd((hd,), torch.float32, g, 0.1)) if norm else None
    kw = (1 + rnd((hd,), torch.float32, g, 0.1)) if norm else None
    positions = torch.randint(0, 300, (n,), generator=g, dtype=torch.int32)
    table = None
    if rope:
        ang = torch.arange(300).float().unsqueeze(1) * torch.pow(
            torch.tensor(10000.0), -2.0 * torch.arange(hd // 2).float() / hd)
        table = (ang.cos(), ang.sin())
    slots = torch.randperm(pages * ps, generator=g)[:n].to(torch.int32)
    slots[5] = -1
    kc = rnd((pages, ps, nkv, hd), dtype, g)
    vc = rnd((pages, ps, nkv, hd), dtype, g)
    ref_qkv, ref_k, ref_v = qkv.clone(), kc.clone(), vc.clone()
    PlainOps().qk_norm_rope_write(ref_qkv, nh, nkv, hd, qw, kw, 1e-6, table, positions, slots,
                                  ref_k, ref_v)
    d_qkv, d_k, d_v = qkv.cuda(), kc.cuda(), vc.cuda()
    ops.qk_norm_rope_write(d_qkv, nh, nkv, hd, qw.cuda() if norm else None,
                           kw.cuda() if norm else None, 1e-6,
                           (table[0].cuda(), table[1].cuda()) if rope else None,
                           positions.cuda(), slots.cuda(), d_k, d_v)
    t = tol(dtype)
    assert torch.allclose(d_qkv[:, :nh * hd].cpu().float(), ref_qkv[:, :nh * hd].float(), **t)
    assert torch.allclose(d_k.cpu().float(), ref_k.float(), **t)
    assert torch.equal(d_v.cpu(), ref_v)


@pytest.mark.parametrize("norm,rope", [(True, True), (False, True), (True, False)])
@pytest.mark.parametrize("sizes", [
    # tokens, heads, kv heads, hidden: an odd number of heads in all (the last tile of 128 rows
    # holds one head), K split over a cluster and not, one token and the most the kernel takes
    (8, 6, 2, 512), (1, 3, 1, 72), (16, 5, 2, 4096), (11, 32, 8, 2048),
])
def test_linear_qk_norm_rope_write(ops, sizes, norm, rope):
    """The q|k|v product with norm, rotation and cache write in its epilogue (bfloat16, head
    size 64, few tokens) against the product followed by the plain norm/rotation/write."""
    n, nh, nkv, hidden = sizes
    hd, ps, pages = 64, 8, 9
    g = torch.Generator().manual_seed(14)
    x = rnd((n, hidden), torch.bfloat16, g)
    w = rnd(((nh + 2 * nkv) * hd, hidden), torch.bfloat16, g, 0.05)
    qw = (1 + rnd((hd,), torch.float32, g, 0.1)) if norm else None
    kw = (1 + rnd((hd,), torch.float32, g, 0.1)) if norm else None
    positions = torch.randint(0, 300, (n,), generator=g, dtype=torch.int32)
    table = None
    if rope:
        ang = torch.arange(300).float().unsqueeze(1) * torch.pow(
            torch.tensor(10000.0), -2.0 * torch.arange(hd // 2).float() / hd)
        table = (ang.cos(), ang.sin())
    slots = torch.randperm(pages * ps, generator=g)[:n].to(torch.int32)
    if n > 5:
        slots[5] = -1
    kc = rnd((pages, ps, nkv, hd), torch.bfloat16, g)
    vc = rnd((pages, ps, nkv, hd), torch.bfloat16, g)
    ref_k, ref_v = kc.clone(), vc.clone()
    ref_qkv = PlainOps().linear_qk_norm_rope_write(x, w, nh, nkv, hd, qw, kw, 1e-6, table,
                                                  positions, slots, ref_k, ref_v)
    dev = lambda t: None if t is None else t.cuda()
    results = []
    fused = ops.fuse_qkv_rope
    try:
        for mode in (True, False):
            ops.fuse_qkv_rope = mode
            d_k, d_v = kc.cuda(), vc.cuda()
            d_qkv = ops.linear_qk_norm_rope_write(
                x.cuda(), w.cuda(), nh, nkv, hd, dev(qw), dev(kw), 1e-6,
                (table[0].cuda(), table[1].cuda()) if rope else None, positions.cuda(),
                slots.cuda(), d_k, d_v)
            ops.check_status()
            results.append((d_qkv[:, :nh * hd].cpu().float(), d_k.cpu().float(), d_v.cpu().float()))
    finally:
        ops.fuse_qkv_rope = fused
    scale = float(ref_qkv.float().abs().max())
    for q_out, k_out, v_out in results:
        # the product's rounding to bfloat16 sits before the norm: a last-bit difference of
        # the product is a last-bit difference of the result
        assert (q_out - ref_qkv[:, :nh * hd].float()).abs().max() <= 2e-2 * scale
        assert (k_out - ref_k.float()).abs().max() <= 2e-2 * scale
        assert (v_out - ref_v.float()).abs().max() <= 2e-2 * scale
    # the slot -1 row wrote nothing; untouched slots are untouched
    written = set(int(s_) for s_ in slots.tolist() if s_ >= 0)
    flat_k = results[0][1].reshape(pages * ps, -1)
    for slot in range(pages * ps):
        if slot not in written:
            assert torch.equal(flat_k[slot], kc.float().reshape(pages * ps, -1)[slot])


def attention_case(dtype, g, q_lens, ctx_lens, nh, nkv, hd, ps, window=None, standout=False):
    """A batch with random pages in a shuffled pool.  With `standout`, one far key of
    every request is made to dominate the softmax of its last query."""
    R = len(q_lens)
    n = sum(q_lens)
    blocks = [-(-c // ps) for c in ctx_lens]
    pages = sum(blocks) + 3
    perm = torch.randperm(pages, generator=g).tolist()
    mb = max(blocks)
    table = torch.full((R, mb), -1, dtype=torch.int32)
    k = 0
    for r in range(R):
        for b in range(blocks[r]):
            table[r, b] = perm[k]
            k += 1
    kc = rnd((pages, ps, nkv, hd), dtype, g)
    vc = rnd((pages, ps, nkv, hd), dtype, g)
    q = rnd((n, (nh + 2 * nkv) * hd), dtype, g)
    q_start = [0]
    for ql in q_lens:
        q_start.append(q_start[-1] + ql)
    token_req = [r for r, ql in enumerate(q_lens) for _ in range(ql)]
    if standout:
        for r in range(R):
            p = ctx_lens[r] - 1
            lo = 0 if window is None else max(0, p - window + 1)
            far = lo + (p - lo) // 7           # a key far from the query, inside the window
            t_last = q_start[r + 1] - 1
            page, slot = int(table[r, far // ps]), far % ps
            for h in range(nh):
                qh = q[t_last, h * hd:(h + 1) * hd].float()
                kc[page, slot, h // (nh // nkv)] = (qh / qh.norm() * 6.0).to(dtype)
    n_decode = 0
    while n_decode < R and q_lens[n_decode] == 1:
        n_decode += 1
    ctx = SimpleNamespace(
        n_tokens=n, n_reqs=R, n_decode=n_decode,
        q_start=torch.tensor(q_start, dtype=torch.int32),
        ctx_lens=torch.tensor(ctx_lens, dtype=torch.int32),
        token_req=torch.tensor(token_req, dtype=torch.int32),
        max_ctx_len=max(ctx_lens), max_q_len=max(q_lens))
    group = SimpleNamespace(block_table=table, max_blocks=mb, page_size=ps, window=window)
    return q, kc, vc, ctx, group


def to_cuda(ns):
    return SimpleNamespace(**{k: (v.cuda() if torch.is_tensor(v) else v)
                              for k, v in vars(ns).items()})


ATTN_CASES = [
    # q_lens, ctx_lens, heads, kv heads, head size, page, window
    ([1, 1, 5, 40], [1, 300, 5, 333], 6, 2, 48, 8, None),
    ([1, 7, 2, 64], [700, 7, 130, 64], 3, 1, 80, 16, None),
    ([1, 1, 9, 33], [290, 17, 100, 260], 8, 2, 16, 16, 37),
    ([3], [515], 4, 4, 128, 32, None),
    # head size 64: the decode kernels that stream pages by TMA (pages of 8, 16, 32, 64)
    ([1, 1, 1, 1, 6], [700, 1, 257, 64, 6], 8, 2, 64, 16, None),
    ([1, 1, 1, 2], [300, 255, 9, 130], 12, 4, 64, 8, 100),
    ([1, 1, 1], [1030, 33, 512], 4, 1, 64, 32, None),
    ([1, 1], [400, 70], 2, 2, 64, 64, 129),
    # 32 query heads on one key/value head: two tiles of 16 packed rows per head group
    ([1, 1, 3], [300, 70, 40], 32, 1, 64, 16, None),
]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", ATTN_CASES)
@pytest.mark.parametrize("standout", [False, True])
def test_paged_attention(ops, dtype, case, standout):
    q_lens, ctx_lens, nh, nkv, hd, ps, window = case
    g = torch.Generator().manual_seed(7)
    q, kc, vc, ctx, group = attention_case(dtype, g, q_lens, ctx_lens, nh, nkv, hd, ps, window,
                                           standout)
    scale = 1.0 / math.sqrt(hd)
    ref = torch.zeros(ctx.n_tokens, nh * hd, dtype=dtype)
    PlainOps().paged_attention(q, nh, nkv, hd, kc, vc, ctx, group, scale, window, ref)
    dq, dk, dv, dctx, dgroup = q.cuda(), kc.cuda(), vc.cuda(), to_cuda(ctx), to_cuda(group)
    t = dict(atol=3e-6, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=2e-2)
    # the dispatching entry (decode kernel for single tokens, prefill kernel for the rest)
    out = torch.full((ctx.n_tokens, nh * hd), float("nan"), dtype=dtype, device="cuda")
    ops.paged_attention(dq, nh, nkv, hd, dk, dv, dctx, dgroup, scale, window, out)
    assert torch.allclose(out.cpu().float(), ref.float(), **t)
    if dtype == torch.bfloat16 and hd == 64:
        # both tensor-core decode kernels by name (the default picks one by the amount of work)
        chosen = ops.decode_kernel
        try:
            for kernel in ("block", "stream"):
                ops.decode_kernel = kernel
                out1 = torch.full((ctx.n_tokens, nh * hd), float("nan"), dtype=dtype, device="cuda")
                ops.paged_attention(dq, nh, nkv, hd, dk, dv, dctx, dgroup, scale, window, out1)
                assert torch.allclose(out1.cpu().float(), ref.float(), **t), kernel
            ops.check_status()
        finally:
            ops.decode_kernel = chosen
    # every token through the general kernel
    out2 = torch.full((ctx.n_tokens, nh * hd), float("nan"), dtype=dtype, device="cuda")
    ops.paged_attention_general(dq, nh, nkv, hd, dk, dv, dctx, dgroup, scale, window, out2)
    assert torch.allclose(out2.cpu().float(), ref.float(), **t)


@pytest.mark.parametrize("reqs,nh,nkv,ps,window", [
    (1, 4, 4, 16, None),          # a request over all runs
    (3, 8, 2, 64, None),
    (31, 4, 2, 16, None),
    (70, 4, 2, 16, None),         # more requests than a warp looks up at once, several in a run
    (70, 6, 2, 8, 129),
    (33, 32, 1, 32, None),        # two teams' warps a key/value head
    (9, 300, 300, 16, 100),       # more heads than a quarter of the warps: several runs a warp
])
def test_decode_stream_runs(ops, reqs, nh, nkv, ps, window):
    """The stream kernel shares the step's tiles out in runs that end anywhere: contexts of all lengths around a
    tile's and a run's edge, empty ones between them.  Bounds as in `test_paged_attention`."""
    hd = 64
    lens = [(1, 64, 700, 65, 3, 128, 129, 1500, 200, 63)[i % 10] if nh < 100 else 60 + 70 * i for i in range(reqs)]
    g = torch.Generator().manual_seed(11)
    q, kc, vc, ctx, group = attention_case(torch.bfloat16, g, [1] * reqs, lens, nh, nkv, hd, ps, window)
    for r in range(5, reqs, 13):
        ctx.ctx_lens[r] = 0
        group.block_table[r] = -1
    ref = torch.zeros(reqs, nh * hd, dtype=torch.bfloat16)
    PlainOps().paged_attention(q, nh, nkv, hd, kc, vc, ctx, group, 0.125, window, ref)
    ref[ctx.ctx_lens == 0] = 0
    out = torch.full((reqs, nh * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    chosen = ops.decode_kernel
    try:
        ops.decode_kernel = "stream"
        ops.paged_attention(q.cuda(), nh, nkv, hd, kc.cuda(), vc.cuda(), to_cuda(ctx), to_cuda(group), 0.125,
                            window, out)
        ops.check_status()
    finally:
        ops.decode_kernel = chosen
    assert torch.allclose(out.cpu().float(), ref.float(), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("nh,nkv", [(1, 1), (32, 8), (8, 1), (12, 1), (20, 1)])
def test_decode_stream_multiplies_all_of_p(ops, nh, nkv):
    """The weights of long runs of keys are multiplied in two bfloat16 parts (2^-17 of each is left out), one query
    head and eight of them with the rest in rows that are free, twelve and sixteen with a product of its own, and
    four heads beyond sixteen: rows of 32 bits against float64.  Powers of two, sums and the products of up to 2,900 keys
    add some 2^-20.  In one part it is 2^-10.  An infinite value stays one."""
    lens, hd = [2900, 2037, 64, 1, 517], 64
    g = torch.Generator().manual_seed(nh)
    q, kc, vc, ctx, group = attention_case(torch.bfloat16, g, [1] * len(lens), lens, nh, nkv, hd, 16)
    page, slot = int(group.block_table[1, 31]), 5
    vc[page, slot, 0, 3] = float("inf")
    out = torch.full((len(lens), nh * hd), float("nan"), device="cuda")
    d_ctx, d_group = to_cuda(ctx), to_cuda(group)
    ops.paged_attention_decode_mma(q.cuda(), nh, nkv, hd, kc.cuda(), vc.cuda(), d_group.block_table, d_ctx.q_start,
                                   d_ctx.ctx_lens, len(lens), max(lens), 16, 0.125, None, out)
    ops.check_status()
    vc[page, slot, 0, 3] = 0
    for r, c in enumerate(lens):
        at = torch.arange(c)
        rows = lambda t: t[group.block_table[r].long()[at // 16], at % 16].double()          # noqa: E731
        k, v = rows(kc), rows(vc)
        for h in range(nh):
            p = torch.softmax(k[:, h * nkv // nh] @ q[r, h * hd:(h + 1) * hd].double() * 0.125, 0)
            got, want = out[r, h * hd:(h + 1) * hd].cpu().double(), p @ v[:, h * nkv // nh]
            if r == 1 and h * nkv // nh == 0:
                assert float(got[3]) == float("inf")
                got[3] = want[3]
            assert float((got - want).norm() / want.norm()) < 2.0 ** -16, (r, h)


EDGE_CASES = [
    # q_len, context, window, page: where the window's first key `lo` of the last (and, for a
    # portion, of the first) query falls
    (1, 356, 100, 16),      # lo = 256: a split, tile and page boundary
    (1, 321, 129, 16),      # lo = 192: a tile boundary inside a split
    (1, 258, 50, 16),       # lo = 208: a page boundary inside a tile
    (1, 356, 100, 64),      # lo = 256 with pages of 64
    (8, 356, 100, 16),      # portion: last query lo = 256
    (8, 363, 100, 16),      # portion: first query lo = 256
    (8, 328, 129, 8),       # portion: first query lo = 192, last 199
    (40, 300, 37, 32),      # portion longer than the window
]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", EDGE_CASES)
def test_window_edge(ops, dtype, case):
    """The first key of a window must count and the key before it must not.  For the first
    and the last query of each request the key at `lo` is made to dominate the softmax, and
    the key at `lo - 1` is made twice as strong again with a value far from all others: a
    kernel that is off by one at the window's edge returns another vector altogether, not a
    slightly different average.  Every attention kernel that can take the case runs it."""
    q_len, clen, window, ps = case
    nh, nkv, hd = 4, 2, 64
    g = torch.Generator().manual_seed(31)
    q_lens, ctx_lens = [q_len, q_len], [clen, clen - 64]
    q, kc, vc, ctx, group = attention_case(dtype, g, q_lens, ctx_lens, nh, nkv, hd, ps, window)
    q_start = ctx.q_start.tolist()
    for r in range(2):
        for t, p in ((q_start[r], ctx_lens[r] - q_len), (q_start[r + 1] - 1, ctx_lens[r] - 1)):
            lo = p - window + 1
            assert lo >= 1
            for h in range(nh):
                qh = q[t, h * hd:(h + 1) * hd].float()
                for key, strength in ((lo, 6.0), (lo - 1, 12.0)):
                    page, slot = int(group.block_table[r, key // ps]), key % ps
                    kc[page, slot, h // (nh // nkv)] = (qh / qh.norm() * strength).to(dtype)
                    if key == lo - 1:
                        vc[page, slot, h // (nh // nkv)] = 50.0
    scale = 1.0 / math.sqrt(hd)
    ref = torch.zeros(ctx.n_tokens, nh * hd, dtype=dtype)
    PlainOps().paged_attention(q, nh, nkv, hd, kc, vc, ctx, group, scale, window, ref)
    wrong = torch.zeros_like(ref)
    PlainOps().paged_attention(q, nh, nkv, hd, kc, vc, ctx, group, scale, window + 1, wrong)
    assert float((wrong.float() - ref.float()).abs().max()) > 10       # the edge decides the result
    dq, dk, dv, dctx, dgroup = q.cuda(), kc.cuda(), vc.cuda(), to_cuda(ctx), to_cuda(group)
    t = dict(atol=3e-5, rtol=1e-4) if dtype == torch.float32 else dict(atol=3e-2, rtol=2e-2)

    def run(label):
        out = torch.full((ctx.n_tokens, nh * hd), float("nan"), dtype=dtype, device="cuda")
        ops.paged_attention(dq, nh, nkv, hd, dk, dv, dctx, dgroup, scale, window, out)
        assert torch.allclose(out.cpu().float(), ref.float(), **t), label

    run("chosen by size")
    if dtype == torch.bfloat16:
        chosen = ops.decode_kernel, ops.prefill_attention
        try:
            if q_len == 1:
                for kernel in ("block", "stream"):
                    ops.decode_kernel = kernel
                    run(kernel)
            else:
                for kernel in ("tcgen05", "mma"):
                    ops.prefill_attention = kernel
                    run(kernel)
            ops.check_status()
        finally:
            ops.decode_kernel, ops.prefill_attention = chosen
    out2 = torch.full((ctx.n_tokens, nh * hd), float("nan"), dtype=dtype, device="cuda")
    ops.paged_attention_general(dq, nh, nkv, hd, dk, dv, dctx, dgroup, scale, window, out2)
    assert torch.allclose(out2.cpu().float(), ref.float(), **t)


@pytest.mark.parametrize("dtype", DTYPES)
def test_paged_attention_padding_rows(ops, dtype):
    """Requests with context 0 are padding: zeros out, nothing read."""
    g = torch.Generator().manual_seed(8)
    q, kc, vc, ctx, group = attention_case(dtype, g, [1, 1, 1], [40, 9, 300], 4, 2, 32, 16)
    ctx.ctx_lens[1] = 0
    group.block_table[1] = -1
    out = torch.full((3, 4 * 32), float("nan"), dtype=dtype, device="cuda")
    ops.paged_attention(q.cuda(), 4, 2, 32, kc.cuda(), vc.cuda(), to_cuda(ctx), to_cuda(group),
                        0.17, None, out)
    assert torch.all(out[1] == 0) and torch.isfinite(out).all()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps,bias", [(3, False), (4, True), (2, True), (5, False), (1, False)])
def test_short_conv(ops, dtype, taps, bias):
    g = torch.Generator().manual_seed(9)
    hidden = 200
    q_lens = [1, 1, 2, 5, 40, 70, 3]
    start = [0, 9, 0, 4, 0, 33, 1]
    slots = [5, 2, 7, 0, 3, 6, -1]
    n = sum(q_lens)
    proj = rnd((n, 3 * hidden), dtype, g)
    filt = rnd((hidden, taps), torch.float32, g, 0.5)
    b_in = rnd((3 * hidden,), torch.float32, g, 0.1) if bias else None
    b_conv = rnd((hidden,), torch.float32, g, 0.1) if bias else None
    state = rnd((8, max(taps - 1, 1), hidden), torch.float32, g)[:, :taps - 1].contiguous()
    q_start = [0]
    for ql in q_lens:
        q_start.append(q_start[-1] + ql)
    ctx = SimpleNamespace(n_reqs=len(q_lens), max_q_len=max(q_lens),
                          q_start=torch.tensor(q_start, dtype=torch.int32),
                          state_slot=torch.tensor(slots, dtype=torch.int32),
                          start_pos=torch.tensor(start, dtype=torch.int32))
    ref, ref_state = torch.empty(n, hidden, dtype=dtype), state.clone()
    PlainOps().short_conv(proj, filt, b_in, b_conv, ref_state if taps > 1 else None, ctx, ref)
    out, d_state = torch.empty(n, hidden, dtype=dtype, device="cuda"), state.cuda()
    ops.short_conv(proj.cuda(), filt.cuda(), b_in.cuda() if bias else None,
                   b_conv.cuda() if bias else None, d_state if taps > 1 else None,
                   to_cuda(ctx), out)
    assert torch.allclose(out.cpu().float(), ref.float(), **tol(dtype))
    if taps > 1:
        assert torch.allclose(d_state.cpu(), ref_state, atol=1e-6, rtol=1e-6)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps,rest", [(3, 2600), (4, 2600), (2, 700), (4, 700), (4, 300)])
def test_short_conv_pieces(ops, dtype, taps, rest):
    """Pieces of 16 tokens in rounds (2,600 tokens of 1,032 channels) and of 4 at once (700, with 4 taps 300), for more requests than
    are looked up at a time and portions around a piece's and a window's length."""
    g = torch.Generator().manual_seed(19)
    hidden = 1032
    q_lens = [1] * 25 + [2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 33, rest, 16, 1]
    n, R = sum(q_lens), len(q_lens)
    start = [(0, 5, 1)[i % 3] for i in range(R)]
    slots = [i if i % 7 else -1 for i in range(R)]
    proj = rnd((n, 3 * hidden), dtype, g)
    filt = rnd((hidden, taps), torch.float32, g, 0.5)
    state = rnd((R, taps - 1, hidden), torch.float32, g)
    q_start = [0]
    for ql in q_lens:
        q_start.append(q_start[-1] + ql)
    ctx = SimpleNamespace(n_reqs=R, max_q_len=max(q_lens), q_start=torch.tensor(q_start, dtype=torch.int32),
                          state_slot=torch.tensor(slots, dtype=torch.int32),
                          start_pos=torch.tensor(start, dtype=torch.int32))
    ref, ref_state = torch.empty(n, hidden, dtype=dtype), state.clone()
    PlainOps().short_conv(proj, filt, None, None, ref_state, ctx, ref)
    out, d_state = torch.full((n, hidden), float("nan"), dtype=dtype, device="cuda"), state.cuda()
    ops.short_conv(proj.cuda(), filt.cuda(), None, None, d_state, to_cuda(ctx), out)
    assert torch.allclose(out.cpu().float(), ref.float(), **tol(dtype))
    assert torch.allclose(d_state.cpu(), ref_state, atol=1e-6, rtol=1e-6)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps", [3, 4])
def test_short_conv_long_portion_equals_short_portions(ops, dtype, taps):
    """A portion of 150 tokens (the kernel for long portions: eight channels a thread, rows
    requested ahead) gives bit for bit what portions of 40 + 63 + 47 tokens give through the
    state (the kernel for short ones), and the same final state."""
    g = torch.Generator().manual_seed(91)
    hidden, n = 328, 150
    proj = rnd((n, 3 * hidden), dtype, g).cuda()
    filt = rnd((hidden, taps), torch.float32, g, 0.5).cuda()
    b_in = rnd((3 * hidden,), torch.float32, g, 0.1).cuda()
    b_conv = rnd((hidden,), torch.float32, g, 0.1).cuda()

    def run(cuts):
        state = torch.zeros(2, taps - 1, hidden, dtype=torch.float32, device="cuda")
        out = torch.empty(n, hidden, dtype=dtype, device="cuda")
        pos = 0
        for ql in cuts:
            ctx = SimpleNamespace(n_reqs=1, max_q_len=ql,
                                  q_start=torch.tensor([0, ql], dtype=torch.int32, device="cuda"),
                                  state_slot=torch.tensor([1], dtype=torch.int32, device="cuda"),
                                  start_pos=torch.tensor([pos], dtype=torch.int32, device="cuda"))
            ops.short_conv(proj[pos:pos + ql], filt, b_in, b_conv, state, ctx, out[pos:pos + ql])
            pos += ql
        return out, state

    whole, whole_state = run([n])
    parts, parts_state = run([40, 63, 47])
    assert torch.equal(whole, parts)
    assert torch.equal(whole_state, parts_state)
    ref = torch.empty(n, hidden, dtype=dtype)
    ref_state = torch.zeros(2, taps - 1, hidden)
    ctx = SimpleNamespace(n_reqs=1, max_q_len=n, q_start=torch.tensor([0, n], dtype=torch.int32),
                          state_slot=torch.tensor([1], dtype=torch.int32),
                          start_pos=torch.tensor([0], dtype=torch.int32))
    PlainOps().short_conv(proj.cpu(), filt.cpu(), b_in.cpu(), b_conv.cpu(), ref_state, ctx, ref)
    assert torch.allclose(whole.cpu().float(), ref.float(), **tol(dtype))
    assert torch.allclose(whole_state.cpu(), ref_state, atol=1e-6, rtol=1e-6)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps", [2, 3, 4])
def test_short_conv_state_of_short_portions(ops, dtype, taps):
    """Many portions of one to five tokens over four steps: a piece of a portion must not see the state that another
    piece has moved on (a piece shorter than the window would, now and then)."""
    g = torch.Generator().manual_seed(23)
    hidden, R = 2048, 60
    filt = rnd((hidden, taps), torch.float32, g, 0.5)
    ref_state = rnd((R, taps - 1, hidden), torch.float32, g)
    state = ref_state.cuda()
    for step in range(4):
        q_lens = [1 + (i * 7 + step * 3) % 5 for i in range(R)]
        q_start = [0]
        for ql in q_lens:
            q_start.append(q_start[-1] + ql)
        n = q_start[-1]
        ctx = SimpleNamespace(n_reqs=R, max_q_len=max(q_lens), q_start=torch.tensor(q_start, dtype=torch.int32),
                              state_slot=torch.arange(R, dtype=torch.int32),
                              start_pos=torch.full((R,), 9, dtype=torch.int32))
        proj = rnd((n, 3 * hidden), dtype, g)
        ref = torch.empty(n, hidden, dtype=dtype)
        PlainOps().short_conv(proj, filt, None, None, ref_state, ctx, ref)
        out = torch.empty(n, hidden, dtype=dtype, device="cuda")
        ops.short_conv(proj.cuda(), filt.cuda(), None, None, state, to_cuda(ctx), out)
        assert torch.allclose(out.cpu().float(), ref.float(), **tol(dtype))
        assert torch.allclose(state.cpu(), ref_state, atol=1e-5, rtol=1e-5)


def test_argmax_first_maximum_and_nan(ops):
    x = torch.randn(5, 1003)
    x[0, 17] = x[0, 900] = 9.0                 # tie: the first wins
    x[1, :] = float("-inf")                    # nothing above -inf: 0
    x[2, 3] = float("nan")
    x[2, 500] = 8.0
    x[3, 1002] = 50.0                          # the last element of a ragged row
    ref = PlainOps().argmax(x)
    out = ops.argmax(x.cuda()).cpu()
    assert out.tolist() == ref.tolist()
    assert out[0] == 17 and out[1] == 0 and out[2] == 500 and out[3] == 1002


@pytest.mark.parametrize("top_p", [1.0, 0.9, 0.3])
def test_sample_matches_definition(ops, top_p):
    g = torch.Generator().manual_seed(11)
    vocab, rows = 1003, 64
    logits = torch.randn(rows, vocab, generator=g) * 3
    temp = torch.full((rows,), 0.8)
    temp[5] = 0.0                               # a greedy row among sampled ones
    tp = torch.full((rows,), top_p)
    seed = torch.arange(rows, dtype=torch.int64) * 7 + 3
    counter = torch.arange(rows, dtype=torch.int64)
    out = ops.sample(logits.cuda(), temp.cuda(), tp.cuda(), seed.cuda(), counter.cuda()).cpu()
    differ = []
    for m in range(rows):
        want = sample_row(logits[m], float(temp[m]), top_p, int(seed[m]), int(counter[m]))
        if int(out[m]) != want:
            differ.append((m, int(out[m]), want))
    # float32 sums against the definition's float64 sums can move a draw that falls
    # within rounding of a boundary to the neighbouring token; that is rare
    assert len(differ) <= 1, differ
    assert int(out[5]) == int(torch.argmax(logits[5]))


@pytest.mark.parametrize("vocab", [1003, 20000, 65536, 73728, 80000])
def test_sample_on_chip_and_from_memory(ops, vocab):
    """The kernel that keeps a row's probabilities in registers and shared memory and the one
    that re-reads the logits in every pass: rows that fit registers alone, registers and
    shared memory, a row that fills the first kernel to its limit, and (80,000) rows too long
    for it, which then is not used.  They add in different orders, so a draw within float32
    rounding of a boundary may go to the neighbouring kept token: at most one row in twelve may
    differ, and both must follow the definition (float64) with the same allowance."""
    g = torch.Generator().manual_seed(vocab)
    rows = 12
    logits = (torch.randn(rows, vocab, generator=g) * 4)
    temp = 0.5 + torch.rand(rows, generator=g)
    temp[7] = 0.0                                   # a greedy row
    tp = torch.tensor([1.0, 0.95, 0.9, 0.5, 0.3, 0.05] * 2)
    seed = torch.arange(rows, dtype=torch.int64) * 13 + 1
    counter = torch.arange(rows, dtype=torch.int64)
    outs = []
    try:
        for mode in (1, 0):
            ops.lib.rv_sample_set_onchip(mode)
            outs.append(ops.sample(logits.cuda(), temp.cuda(), tp.cuda(), seed.cuda(),
                                   counter.cuda()).cpu())
    finally:
        ops.lib.rv_sample_set_onchip(1)
    assert int((outs[0] != outs[1]).sum()) <= 1
    want = torch.tensor([sample_row(logits[m], float(temp[m]), float(tp[m]), int(seed[m]),
                                    int(counter[m])) for m in range(rows)], dtype=torch.int32)
    for got in outs:
        assert int((got != want).sum()) <= 1, (got.tolist(), want.tolist())
        assert int(got[7]) == int(torch.argmax(logits[7]))


@pytest.mark.parametrize("rows,vocab", [
    # one, two, four and eight blocks a row at their limits; the steps in values a thread; many rows
    # (32 values a thread before a further block); the longest row a cluster takes and one more
    (3, 4096), (3, 4097), (3, 16385), (3, 32769), (3, 49153), (3, 81921), (3, 131072), (3, 131073),
    (33, 5), (33, 8193), (40, 65536)])
def test_sample_cluster_edges(ops, rows, vocab):
    """The kernel that spreads a row over a cluster against the one that re-reads the logits: at
    most one draw in a call may fall within float32 rounding of a boundary (the sums are taken in
    another order).  Rows whose outcome rounding cannot move agree exactly: one probability that
    outweighs the others, the value tied everywhere with top-p 0, greedy rows, NaN and infinities."""
    g = torch.Generator().manual_seed(vocab)
    logits = torch.randn(rows, vocab, generator=g) * 4
    tp = torch.tensor([0.95, 0.9999, 0.5])[torch.arange(rows) % 3].clone()
    temp = torch.full((rows,), 0.8)
    cases = []
    if rows > 3:
        logits[3, vocab // 2] = 400.0                          # everything on one token
        logits[4] = 1.0                                        # ties with top-p 0: all of them are kept
        tp[4] = 0.0
        logits[5, vocab // 3] = float("nan")
        logits[6] = float("-inf")
        logits[7, 1] = float("inf")
        logits[8, 2:] = float("-inf")
        temp[9] = 0.0                                          # greedy, with a tie and a NaN
        logits[9, 0] = float("nan")
        logits[9, [1, vocab - 1]] = 1000.0
        cases = [3, 6, 7, 9]
    seed = torch.arange(rows, dtype=torch.int64) * 13 + 1
    counter = torch.arange(rows, dtype=torch.int64)
    outs = []
    try:
        for mode in (1, 0):
            ops.lib.rv_sample_set_onchip(mode)
            outs.append(ops.sample(logits.cuda(), temp.cuda(), tp.cuda(), seed.cuda(),
                                   counter.cuda()).cpu())
    finally:
        ops.lib.rv_sample_set_onchip(1)
    assert int((outs[0] != outs[1]).sum()) <= 1, (outs[0].tolist(), outs[1].tolist())
    for m in cases:
        assert int(outs[0][m]) == int(outs[1][m])
    if rows > 3:
        assert int(outs[0][9]) == 1
        assert int(outs[0][3]) == vocab // 2


def test_sample_frequencies(ops):
    """Draws over many counters follow softmax(logits / T)."""
    logits = torch.tensor([[2.0, 1.0, 0.0, -1.0, 0.5]])
    n = 4000
    L = logits.repeat(n, 1).cuda()
    out = ops.sample(L, torch.full((n,), 0.7).cuda(), torch.ones(n).cuda(),
                     torch.full((n,), 1234, dtype=torch.int64).cuda(),
                     torch.arange(n, dtype=torch.int64).cuda()).cpu()
    freq = torch.bincount(out.long(), minlength=5).double() / n
    p = torch.softmax(logits[0].double() / 0.7, 0)
    assert (freq - p).abs().max() < 0.03


GEMM_SHAPES = [
    # M, N, K: token counts around the padding steps, widths that are no multiple of the
    # 128-row tile or the 64-element stage, K split over many blocks and not split at all
    (1, 128, 64), (3, 200, 72), (8, 2048, 2048), (16, 6144, 2048), (17, 1000, 520),
    (64, 2048, 8192), (100, 384, 96), (128, 16384, 256), (200, 640, 1096), (256, 130, 2048),
]


@pytest.mark.parametrize("M,N,K", GEMM_SHAPES)
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_tcgen05(ops, M, N, K, out_dtype):
    g = torch.Generator().manual_seed(12)
    x = rnd((M, K), torch.bfloat16, g)
    w = rnd((N, K), torch.bfloat16, g, 0.05)
    # one entry of x and w made large: a wrong tile, swizzle or K offset cannot hide
    x[M // 2, K // 3] = 40.0
    w[N // 5, K // 3] = 3.0
    ref = x.double() @ w.double().t()
    for _ in range(2):                            # twice: the tickets must be back at zero
        y = ops.linear_tcgen05(x.cuda(), w.cuda(), out_dtype)
        ops.check_status()
        err = (y.double().cpu() - ref).abs().max() / ref.abs().max()
        assert err <= (2e-5 if out_dtype == torch.float32 else 5e-3), float(err)
    # the same numbers whatever rows share the batch: row 0 alone
    y1 = ops.linear_tcgen05(x[:1].contiguous().cuda(), w.cuda(), torch.float32)
    yM = ops.linear_tcgen05(x.cuda(), w.cuda(), torch.float32)
    assert torch.equal(y1[0], yM[0])



@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (3, 200, 72), (8, 2048, 2048), (16, 6144, 2048),
                                   (5, 2048, 8192), (16, 1000, 520), (64, 2048, 8192)])
def test_gemm_tiled_weights(ops, M, N, K):
    """With the weight matrix laid out tile by tile (contiguous bulk copies of two K blocks a
    stage) and with tensor-map boxes of the row-major matrix the MMAs run over the same values in
    the same order: bit-identical results, for tiles and K blocks that the matrix fills only
    partly, K split over a cluster and not; the tiled copy is made once per matrix."""
    g = torch.Generator().manual_seed(13)
    x = rnd((M, K), torch.bfloat16, g).cuda()
    w = rnd((N, K), torch.bfloat16, g, 0.05).cuda()
    was = ops.gemm_tiled
    try:
        ops.gemm_tiled = True
        a = ops.linear_tcgen05(x, w, torch.float32)
        copies = len(ops._tiled)
        a2 = ops.linear_tcgen05(x, w, torch.float32)
        assert len(ops._tiled) == copies                      # the same copy again
        ops.gemm_tiled = False
        b = ops.linear_tcgen05(x, w, torch.float32)
    finally:
        ops.gemm_tiled = was
    ops.check_status()
    assert torch.equal(a, b) and torch.equal(a, a2)
    ref = x.double() @ w.double().t()
    assert float((a.double() - ref).abs().max() / ref.abs().max()) <= 2e-5


@pytest.mark.parametrize("M,N,K", [
    # one to twenty row tiles, columns that fill no tile, K that fills no step (and no split of K), K split over one to
    # eight blocks
    (1, 256, 256), (8, 300, 1028), (9, 2048, 260), (16, 70000, 512), (24, 4608, 1536), (32, 1001, 2052),
    (40, 520, 4096), (48, 640, 1024), (56, 257, 3000), (64, 6144, 256), (65, 1536, 6912), (131, 2048, 516),
    (160, 333, 1540)])
def test_gemm_f32(ops, M, N, K):
    """The float32 product against float64.  Each output is up to sixteen sums (even and odd k, eight
    parts of K) of at most K / 2 fused multiply-adds: its error is below (K / 2 + 16) 2^-24 of the sum of
    the terms' magnitudes, whatever the order; the sums here are far inside that."""
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, K, generator=g)
    w = torch.randn(N, K, generator=g) * 0.05
    x[M // 2, K // 3] = 40.0
    w[N // 5, K // 3] = 3.0
    xd, wd = x.cuda(), w.cuda()
    y = torch.empty(M, N, device="cuda")
    assert ops.lib.rv_gemm_f32(_ptr(xd), _ptr(wd), _ptr(y), c_int(M), c_int(N), c_int(K), ops._stream()) == 0
    ref = x.double() @ w.double().t()
    bound = (K / 2 + 16) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    assert bool(((y.double().cpu() - ref).abs() <= bound).all())
    assert float((y.double().cpu() - ref).norm() / ref.norm()) < 1e-6


@pytest.mark.parametrize("M,N,K,launches", [
    # the split product, from K 512 and 256 columns on (two launches); the other kernel's few sizes (one), and beyond
    # each of their ends; the library (none)
    (40, 256, 512, 2), (8, 9216, 1024, 1), (9, 9216, 1024, 2), (8, 9216, 1020, 2), (8, 8188, 1024, 2), (8, 10244, 1024, 2),
    (1, 8192, 2048, 1), (1, 8192, 2052, 2), (8, 256, 508, 0), (8, 252, 512, 0)])
def test_float32_products_by_size(ops, M, N, K, launches):
    """Which kernel a float32 product takes; the bound is `test_gemm_f32`'s, the widest of the three."""
    g = torch.Generator().manual_seed(K)
    x, w = torch.randn(M, K, generator=g).cuda(), torch.randn(N, K, generator=g).cuda()
    before = ops.launches
    y = ops.linear(x, w)
    assert ops.launches == before + launches
    ref = x.double() @ w.double().t()
    ops.check_status()
    assert bool(((y.double() - ref).abs() <= (K / 2 + 16) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())).all())


@pytest.mark.parametrize("M,N,K", [
    # one chunk of K and a K that fills none, columns that fill no tile, every number of rows' tiles from
    # one row to a full tile and one row more, K shared by one to eight blocks, two and three row tiles,
    # rows that are split in portions
    (1, 256, 768), (15, 300, 4), (17, 130, 100), (33, 257, 772), (49, 129, 3000), (65, 4608, 1536), (96, 128, 8192),
    (113, 1000, 1028), (128, 13824, 768), (131, 1536, 6912), (160, 1030, 2048), (161, 1024, 800), (400, 2048, 2052),
    (1000, 260, 16384)])
def test_gemm_f32_split(ops, M, N, K):
    """The float32 product from bfloat16 parts against float64.  The product of parts that is left out is below
    2^-30 of a term.  A chunk's sixteen sums lose up to two units in the last place each (2^-23), the K / 32 chunks
    and eight blocks half a unit each: (K / 32 + 64) 2^-24 of the sum of the terms' magnitudes, whatever the order."""
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, K, generator=g)
    w = torch.randn(N, K, generator=g) * 0.05
    x[M // 2, K // 3] = 40.0
    w[N // 5, K // 3] = 3.0
    x, w = x.cuda(), w.cuda()
    before = ops.launches
    y = ops._linear_split(x, w)
    assert ops.launches == before + (4 if K > 16000 else 2)       # two kernels a portion of rows
    if ops._split_better(M, N, K):
        assert torch.equal(y, ops.linear(x, w))
    ref = x.double() @ w.double().t()
    ops.check_status()
    bound = (K / 32 + 64) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    assert bool(((y.double() - ref).abs() <= bound).all())
    assert float((y.double() - ref).norm() / ref.norm()) < 5e-7


@pytest.mark.parametrize("M,N,K", [(5, 300, 1028), (161, 1024, 800)])
def test_gemm_f32_split_of_what_is_not_finite(ops, M, N, K):
    """Infinite values, values that are none and values whose first part rounds up to infinity reach the
    outputs that they belong to, as multiply-adds bring them there, and no others."""
    g = torch.Generator().manual_seed(M)
    x = torch.randn(M, K, generator=g)
    w = torch.randn(N, K, generator=g) * 0.05
    x[0, 7], x[1, 30], x[2, K - 1], x[3, 5] = float("inf"), float("nan"), 3.4028234e38, -float("inf")
    w[4], w[5, 7], w[6, 3], w[7, 9] = 0.0, 0.0, float("inf"), float("nan")
    w[:, K - 1] *= 1e-3
    x, w = x.cuda(), w.cuda()
    y = ops._linear_split(x, w)
    ops.check_status()
    ref = (x.double() @ w.double().t()).float()
    assert torch.equal(torch.isnan(y), torch.isnan(ref))
    assert torch.equal(torch.isinf(y) & (y > 0), torch.isinf(ref) & (ref > 0))
    fin = torch.isfinite(ref)
    bound = (K + 64) * 2.0 ** -24 * (x.nan_to_num(0, 0, 0).double().abs() @ w.nan_to_num(0, 0, 0).double().abs().t())
    assert bool(((y.double() - ref.double()).abs() <= bound)[fin].all())


@pytest.mark.parametrize("M,N,K", [(20, 300, 1028), (161, 1024, 800)])
def test_gemm_f32_split_holds_all_bits(ops, M, N, K):
    """What float32 multiply-adds give without any rounding is that here too: values beside a power of two, in either
    operand, and whole numbers whose sums stay below 2^24.  Operands near the ends of float32's range lose no more than
    others (the bound is `test_gemm_f32_split`'s)."""
    g = torch.Generator().manual_seed(K)
    full = lambda *s: (torch.randint(1 << 23, 1 << 24, s, generator=g) * 2.0 ** -23 *           # noqa: E731
                       (1 - 2 * torch.randint(0, 2, s, generator=g))).float().cuda()
    x, w = torch.zeros(M, K, device="cuda"), torch.zeros(N, K, device="cuda")
    at, power = torch.randint(0, K, (M,), generator=g), torch.randint(-20, 20, (M,), generator=g)
    x[torch.arange(M), at] = (2.0 ** power.double()).float().cuda()
    wide = full(N, K)
    assert torch.equal(ops._linear_split(x, wide), wide[:, at].t() * x[torch.arange(M), at][:, None])
    at = torch.randint(0, K, (N,), generator=g)
    w[torch.arange(N), at] = 1.0
    wide = full(M, K)
    assert torch.equal(ops._linear_split(wide, w), wide[:, at])
    x = torch.randint(-4095, 4096, (M, K), generator=g).cuda().float()
    w = torch.randint(-3, 4, (N, K), generator=g).cuda().float()
    assert torch.equal(ops._linear_split(x, w).double(), x.double() @ w.double().t())
    for ex, ew in ((-108, 40), (-112, 0), (-60, -60), (-125, 9), (90, 25)):          # (4 K 2^115 is no overflow)
        x, w = full(M, K) * 2.0 ** ex, full(N, K) * 2.0 ** ew
        ref = x.double() @ w.double().t()
        bound = (K / 32 + 64) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
        # (an output below 2^-126 has float32's last place, 2^-149, and so has every multiply-add there)
        assert bool(((ops._linear_split(x, w).double() - ref).abs() <= bound + K * 2.0 ** -149).all()), (ex, ew)
    ops.check_status()


@pytest.mark.parametrize("M,N,K", [(5, 4608, 1536), (64, 1536, 6912)])
def test_gemm_f32_of_a_matrix_made_just_before(ops, M, N, K):
    """The matrix may be what the launch before writes: a bfloat16 one is cast for float32 rows, and
    a caller may update its matrix between two products.  Every product is of the new values; the
    bound is the one above, of the terms' magnitudes."""
    g = torch.Generator().manual_seed(M)
    x = torch.randn(M, K, generator=g).cuda()
    w16 = [(torch.randn(N, K, generator=g) * 0.05).bfloat16().cuda() for _ in range(2)]
    bound = [(K / 2 + 16) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t()) for w in w16]
    w32 = torch.empty(N, K, device="cuda")
    ys = []
    for i in range(12):
        ys.append((i & 1, ops.linear(x, w16[i & 1])))          # cast, then multiplied
        w32.copy_(w16[i & 1])
        ys.append((i & 1, ops.linear(x, w32)))
        ops.add_bias(w32, torch.ones(K, device="cuda"))        # a launch that lets the next one in early
        ops.add_bias(w32, torch.full((K,), -1.0, device="cuda"))
    for i, y in ys:
        assert bool(((y.double() - x.double() @ w16[i].double().t()).abs() <= bound[i]).all())
    w32.zero_()
    ops.add_bias(w32, torch.ones(K, device="cuda"))
    y = ops.linear(x, w32)
    assert bool(((y.double() - x.double().sum(1, keepdim=True)).abs() <=
                 (K / 2 + 16) * 2.0 ** -24 * x.double().abs().sum(1, keepdim=True)).all())


PREFILL_CASES = [
    # q_lens, ctx_lens, heads, kv heads, head size, page size, window.  Head size 64: the
    # tcgen05 kernel (128 rows = tokens x heads of a group, tiles of 64 keys): group sizes
    # that do and do not divide 128, one head per group, portions that start in the middle of
    # a context and end inside a tile or a page, several tiles, a window, every page size.
    ([40], [40], 4, 1, 64, 16, None),
    ([128, 3], [128, 3], 8, 2, 64, 16, None),
    ([130], [130], 8, 2, 64, 16, None),
    ([70, 5, 200], [170, 5, 500], 12, 4, 64, 8, None),
    ([33, 64], [400, 64], 6, 2, 64, 32, 100),
    ([50, 2], [50, 700], 3, 3, 64, 64, None),
    ([300], [1000], 5, 1, 64, 16, 257),
    ([257], [257], 1, 1, 64, 16, None),
    ([20, 9], [90, 9], 32, 1, 64, 16, None),      # 4 query tokens per block of 128 rows
    ([15], [75], 7, 1, 64, 8, None),              # 18 tokens x 7 heads = 126 rows, 2 unused
    # few blocks and long contexts: the key tiles of a block are shared out over several blocks
    # and merged (4 parts; 3 parts of which the shorter request fills only some; with a window)
    ([40], [2000], 8, 2, 64, 16, None),
    ([100, 7], [3000, 900], 4, 4, 64, 32, None),
    ([64], [1800], 8, 2, 64, 16, 700),
    ([30], [8100], 8, 2, 64, 16, None),           # 16 parts
    # with a window, shared out by the tiles within it: many blocks; a window of fewer than four tiles
    ([100, 60], [900, 1000], 32, 8, 64, 16, 300),
    ([40], [2000], 8, 2, 64, 16, 200),
]


@pytest.mark.parametrize("case", PREFILL_CASES)
@pytest.mark.parametrize("standout", [False, True])
def test_prefill_attention_kernels(ops, case, standout):
    """Prompt portions through each bfloat16 prefill kernel by name."""
    q_lens, ctx_lens, nh, nkv, hd, ps, window = case
    g = torch.Generator().manual_seed(21)
    q, kc, vc, ctx, group = attention_case(torch.bfloat16, g, q_lens, ctx_lens, nh, nkv, hd, ps,
                                           window, standout)
    scale = 1.0 / math.sqrt(hd)
    ref = torch.zeros(ctx.n_tokens, nh * hd, dtype=torch.bfloat16)
    PlainOps().paged_attention(q, nh, nkv, hd, kc, vc, ctx, group, scale, window, ref)
    dq, dk, dv, dctx, dgroup = q.cuda(), kc.cuda(), vc.cuda(), to_cuda(ctx), to_cuda(group)
    chosen = ops.prefill_attention
    try:
        for kernel in ("tcgen05", "mma", "simt"):
            ops.prefill_attention = kernel
            out = torch.full((ctx.n_tokens, nh * hd), float("nan"), dtype=torch.bfloat16,
                             device="cuda")
            ops.paged_attention(dq, nh, nkv, hd, dk, dv, dctx, dgroup, scale, window, out)
            ops.check_status()
            assert torch.allclose(out.cpu().float(), ref.float(), atol=2e-2, rtol=2e-2), kernel
    finally:
        ops.prefill_attention = chosen


@pytest.mark.parametrize("same", [False, True])
@pytest.mark.parametrize("case", [c for c in PREFILL_CASES if max(c[1]) > 64])
def test_prefill_attention_head_size_128(ops, case, same):
    """Head size 128 (two halves of 64 dimensions a tile), with values of their own and with values
    that are the keys (one page tensor under both names), through the default choice; with a sink
    per head.  The same cases and bound as at head size 64."""
    q_lens, ctx_lens, nh, nkv, _, ps, window = case
    hd = 128
    g = torch.Generator().manual_seed(23)
    q, kc, vc, ctx, group = attention_case(torch.bfloat16, g, q_lens, ctx_lens, nh, nkv, hd, ps,
                                           window, True)
    vc = kc if same else vc
    sinks = torch.randn(nh, generator=g)
    scale = 1.0 / math.sqrt(hd)
    ref = torch.zeros(ctx.n_tokens, nh * hd, dtype=torch.bfloat16)
    PlainOps().paged_attention(q, nh, nkv, hd, kc, vc, ctx, group, scale, window, ref, sinks=sinks)
    dk = kc.cuda()
    dv = dk if same else vc.cuda()
    out = torch.full((ctx.n_tokens, nh * hd), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.paged_attention(q.cuda(), nh, nkv, hd, dk, dv, to_cuda(ctx), to_cuda(group), scale, window,
                        out, sinks=sinks.cuda())
    ops.check_status()
    assert ("tcgen05", 128, same) in ops._attn_libs
    assert torch.allclose(out.cpu().float(), ref.float(), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("hd,same", [(64, False), (128, False), (128, True)])
@pytest.mark.parametrize("q_lens,ctx_lens,ps", [([70], [70], 16), ([33, 130], [433, 130], 64), ([20], [1994], 8),
                                                ([300, 5, 66], [300, 90, 2000], 32)])
def test_prefill_attention_slots_beyond_the_context(ops, hd, same, q_lens, ctx_lens, ps):
    """The last page's slots beyond a request's context may hold what another request left there, a
    NaN or an infinity: the outputs are the same as with zeros there, to the bit."""
    g = torch.Generator().manual_seed(hd)
    q, kc, vc, ctx, group = attention_case(torch.bfloat16, g, q_lens, ctx_lens, 8, 2, hd, ps)
    outs = []
    for junk in (0.0, float("nan"), float("inf")):
        k, v = kc.clone(), (None if same else vc.clone())
        for r, c in enumerate(ctx_lens):
            last = int(group.block_table[r, (c - 1) // ps])
            for t in (k, v):
                if t is not None:
                    t.view(-1, ps, 2, hd)[last, (c - 1) % ps + 1:] = junk
        dk = k.cuda()
        dv = dk if same else v.cuda()
        out = torch.empty(sum(q_lens), 8 * hd, dtype=torch.bfloat16, device="cuda")
        ops.paged_attention(q.cuda(), 8, 2, hd, dk, dv, to_cuda(ctx), to_cuda(group), hd ** -0.5, None, out)
        outs.append(out)
    ops.check_status()
    assert ("tcgen05", hd, same) in ops._attn_libs and bool(torch.isfinite(outs[0]).all())
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("same", [False, True])
@pytest.mark.parametrize("lens", [[80], [33, 130]])
def test_prefill_attention_head_size_128_rounds_alike(ops, lens, same):
    """The two prompt kernels round the same probabilities (a row's largest is exactly 1) and divide by
    the sum of the rounded values.  What is left is the order of float32 sums, some 1e-6, which moves
    some 1e-3 of the bfloat16 roundings by 2^-8: sqrt(1e-3) 2^-8 = 1.2e-4 together, and four times that
    is the bound.  Other offsets, or a sum of unrounded values, give 3e-3."""
    g = torch.Generator().manual_seed(24)
    q, kc, vc, ctx, group = attention_case(torch.bfloat16, g, lens, lens, 8, 2, 128, 16)
    k = kc.cuda()
    v = k if same else vc.cuda()
    outs, chosen = [], ops.prefill_attention
    try:
        for kernel in ("tcgen05", "mma"):
            ops.prefill_attention = kernel
            out = torch.empty(sum(lens), 8 * 128, dtype=torch.bfloat16, device="cuda")
            ops.paged_attention(q.cuda(), 8, 2, 128, k, v, to_cuda(ctx), to_cuda(group), 128 ** -0.5, None, out)
            outs.append(out.double())
        ops.check_status()
    finally:
        ops.prefill_attention = chosen
    assert float((outs[0] - outs[1]).norm() / outs[1].norm()) < 4.9e-4


@pytest.mark.parametrize("head_dim,same,blocks", [(64, False, 3), (128, False, 2), (128, True, 2)])
def test_prefill_attention_blocks_a_multiprocessor(ops, head_dim, same, blocks):
    """As many blocks' shared memory fits a multiprocessor as the kernel's bounds are set for, so
    that one block's softmax runs beside another's copies and products."""
    need = getattr(ops._attn5_lib(head_dim, same),
                   f"rv_paged_attention_prefill_tcgen05_shared_bytes_hd{head_dim}")()
    # a block's memory is given out in pieces of 128 bytes
    assert 0 < blocks * (-(-need // 128) * 128) <= \
        torch.cuda.get_device_properties(0).shared_memory_per_multiprocessor


CLUSTERS = [
    # whole prompts in clusters of four and of two, just over one part's tiles; parts that become clusters
    # of four, three and two; a second request of which most blocks have no tokens; blocks of the
    # cluster without tiles (fewer tiles than blocks); a window; latent rows; and one of many blocks, which takes none
    (64, 16, 8, [449], [449], None, 4), (64, 16, 8, [700], [700], None, 4), (64, 16, 8, [1000], [1000], None, 2),
    (64, 32, 8, [512], [1212], None, 2), (64, 32, 8, [128], [1128], None, 3), (64, 32, 8, [256], [2256], None, 4),
    (64, 16, 8, [300, 700], [300, 700], None, 2), (64, 16, 8, [700, 3], [700, 700], None, 2), (64, 16, 8, [1000], [1500], 700, 2),
    (128, 16, 1, [1000], [1000], None, 2), (128, 16, 1, [512], [2012], None, 4), (128, 32, 8, [256], [2256], None, 4),
    (128, 16, 1, [1000], [1500], 640, 2), (64, 32, 8, [1000, 1000], [1000, 1000], None, 1)]


def _cluster_of(ops, hd, heads, kv, lens, ctxs, window):
    fn = getattr(ops._attn5_lib(hd, kv == 1), f"rv_paged_attention_prefill_tcgen05_cluster_hd{hd}")
    return fn(*(c_int(v) for v in (sum(lens), len(lens), max(lens), max(ctxs), heads, kv, window or 0, ops._sm_count)))


def test_prefill_attention_forced_parts_take_no_cluster():
    """RVLLM_PREFILL_SPLIT=1 shares nothing out, other numbers through memory."""
    code = ("import sys; sys.path.insert(0, 'tests'); import test_gpu_kernels as t; from rvllm_b200.kernels import cuda_ops; "
            "print(*[t._cluster_of(cuda_ops(), *c[:-1]) for c in t.CLUSTERS])")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for parts in ("1", "3"):
        out = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, RVLLM_PREFILL_SPLIT=parts),
                             capture_output=True, text=True, timeout=300)
        assert out.returncode == 0, out.stderr[-2000:]
        assert out.stdout.split() == ["1"] * len(CLUSTERS)


@pytest.mark.parametrize("hd,heads,kv,lens,ctxs,window,cluster", CLUSTERS)
def test_prefill_attention_in_clusters(ops, hd, heads, kv, lens, ctxs, window, cluster):
    """Blocks that share a block's key tiles and meet in distributed shared memory, against float64.  P and
    the outputs are rounded to bfloat16 (2^-9 of each at the most, of both signs): 2^-8 of the outputs' norm."""
    g = torch.Generator().manual_seed(sum(lens) + hd)
    assert _cluster_of(ops, hd, heads, kv, lens, ctxs, window) == cluster
    q, kc, vc, ctx, group = attention_case(torch.bfloat16, g, lens, ctxs, heads, kv, hd, 16)
    same = kv == 1
    if same:
        vc = kc
    N = sum(lens)
    k, v = kc.cuda(), None
    v = k if same else vc.cuda()
    out = torch.empty(N, heads * hd, dtype=torch.bfloat16, device="cuda")
    sinks = torch.randn(heads, generator=g).cuda() if window else None
    ops.paged_attention(q.cuda(), heads, kv, hd, k, v, to_cuda(ctx), to_cuda(group), hd ** -0.5, window, out, sinks=sinks)
    ops.check_status()
    a = 0
    for r, (n, c) in enumerate(zip(lens, ctxs)):
        at = torch.arange(c)
        page = group.block_table[r].cpu().long()[at // 16]
        rows = lambda t: t.cpu()[page, at % 16].double().cuda()                          # noqa: E731
        kk, vv = rows(kc), rows(vc)
        qq = q[a:a + n, :heads * hd].view(n, heads, hd).double().cuda()
        pos = torch.arange(c - n, c, device="cuda")[:, None]
        key = torch.arange(c, device="cuda")[None]
        hidden = (key > pos) | (key <= pos - window if window else key < 0)
        for h in range(heads):
            s = (qq[:, h] @ kk[:, h * kv // heads].T * hd ** -0.5).masked_fill(hidden, -float("inf"))
            if sinks is not None:
                s = torch.cat([s, sinks[h].double().expand(n, 1)], 1)
            w = torch.softmax(s, -1)[:, :c] @ vv[:, h * kv // heads]
            got = out[a:a + n, h * hd:(h + 1) * hd].double()
            assert float((got - w).norm() / w.norm()) < 2.0 ** -8, (r, h)
        a += n


def test_prefill_attention_tcgen05_is_used(ops):
    """The default choice takes the tcgen05 kernel where it applies (its launch is counted by
    its own library) and refuses nothing it cannot do: other head sizes go to the mma kernel."""
    g = torch.Generator().manual_seed(22)
    for hd, expect in ((64, True), (32, False)):
        q, kc, vc, ctx, group = attention_case(torch.bfloat16, g, [20], [20], 4, 2, hd, 16)
        out = torch.empty(20, 4 * hd, dtype=torch.bfloat16, device="cuda")
        assert ops._tcgen05_prefill_ok(q.cuda(), out, 4, 2, hd, 16) is expect
        ops.paged_attention(q.cuda(), 4, 2, hd, kc.cuda(), vc.cuda(), to_cuda(ctx), to_cuda(group),
                            0.2, None, out)
        assert torch.isfinite(out).all()
