"""Kernels at the sizes where their tiles, rings, splits and register rows begin and end, against float64 (or exactly)."""
import ctypes
import os

import pytest
import torch

from jittor_b200 import _capi as C

pytestmark = pytest.mark.gpu


class forced:
    """Environment switches of the kernels' plans, for one block."""

    def __init__(self, **names):
        self.names = {"B200JT_" + k: str(v) for k, v in names.items()}

    def __enter__(self):
        self.old = {k: os.environ.get(k) for k in self.names}
        os.environ.update(self.names)

    def __exit__(self, *exc):
        for k, v in self.old.items():
            os.environ.pop(k) if v is None else os.environ.__setitem__(k, v)


def matmul(a, b, ta, tb, scratch=True):
    c = torch.full((a.shape[1 if ta else 0], b.shape[0 if tb else 1]), float("nan"), dtype=a.dtype, device="cuda")
    args = (C.desc(a), C.desc(b), C.desc(c), int(ta), int(tb))
    size, ptr, ws = C.workspace("b200jt_matmul_workspace", *args)
    C.call("b200jt_matmul", *args, *((ptr, size) if scratch else (None, 0)))
    return c


def product(a, b, ta, tb):
    return (a.double().t() if ta else a.double()) @ (b.double().t() if tb else b.double())


# ---- float32 on the tensor cores (csrc/gemm_f32_tc.cu)
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("pair,bn,splits", [(0, 32, 1), (0, 96, 2), (0, 128, 4), (0, 64, 8), (1, 128, 1), (1, 192, 1), (1, 256, 1)])
@pytest.mark.parametrize("m,k,n", [(1, 32, 1), (127, 257, 65), (129, 545, 130), (300, 97, 513)])
def test_f32_tensor_core_matmul(m, k, n, pair, bn, splits, ta, tb):
    a, b = torch.randn(*((k, m) if ta else (m, k)), device="cuda"), torch.randn(*((n, k) if tb else (k, n)), device="cuda")
    with forced(F32TC=1, F32TC_PAIR=pair, F32TC_BN=bn, F32TC_SPLITS=splits):
        c = matmul(a, b, ta, tb)
    want = product(a, b, ta, tb)
    # per 64 of k four truncated additions, each below 2^-23 of the sum so far, then one rounding per 64 of k; no sum exceeds that of
    # the products' magnitudes
    assert (c.double() - want).norm() <= (4 + k / 128) * 2.0 ** -23 * product(a.abs(), b.abs(), ta, tb).norm()
    assert C.lib.b200jt_device_status() == 0


# Relative to the result, operands of both signs and of one. Truncation loses at most 2^-23 of the sum so far at each of the last four
# additions of a group, 1.25 * 2^-23 of its sum on average where all have one sign; the group sums, up to 64 of them, are rounded to
# nearest, 2^-24 each, in random directions. Without the products of the third parts (2^-18 of an operand) or of the two second
# parts the error for operands of both signs would be 8 to 12 times the bound.
@pytest.mark.parametrize("pair,bn,splits", [(0, 128, 1), (0, 64, 8), (1, 256, 1)])
@pytest.mark.parametrize("k", [64, 257, 1024, 4096])
@pytest.mark.parametrize("sign", ["both", "one"])
def test_f32_tensor_core_matmul_accuracy(sign, k, pair, bn, splits):
    a, b = torch.randn(256, k, device="cuda"), torch.randn(k, 384, device="cuda")
    if sign == "one":
        a, b = a.abs(), b.abs()
    with forced(F32TC=1, F32TC_PAIR=pair, F32TC_BN=bn, F32TC_SPLITS=min(splits, k // 32)):
        c = matmul(a, b, 0, 0)
    want = product(a, b, 0, 0)
    assert (c.double() - want).norm() <= 2.5 * 2.0 ** -23 * want.norm()


@pytest.mark.parametrize("pair,bn,splits", [(0, 96, 1), (0, 128, 4), (1, 256, 1)])
def test_f32_tensor_core_matmul_keeps_all_bits(pair, bn, splits):
    """24 significant bits times powers of two, one to a row or column: nothing is rounded, so nothing may be lost."""
    m, k = 270, 300
    pick = torch.randperm(k, device="cuda")
    scale = torch.ldexp(torch.ones(k, device="cuda"), torch.randint(-20, 20, (k,), device="cuda")) * torch.randint(0, 2, (k,), device="cuda").sub(0.5).sign()
    p = torch.zeros(k, k, device="cuda")
    p[pick, torch.arange(k, device="cuda")] = scale
    v = torch.randn(m, k, device="cuda")
    with forced(F32TC=1, F32TC_PAIR=pair, F32TC_BN=bn, F32TC_SPLITS=splits):
        assert torch.equal(matmul(v, p, 0, 0), v[:, pick] * scale)
        assert torch.equal(matmul(p, v, 1, 1), (v[:, pick] * scale).t())


def test_f32_tensor_core_matmul_range():
    """Subnormal and huge operands, overflow, infinities and NaN come out as from float32 arithmetic."""
    m, k, n = 130, 200, 140
    a, b = torch.randn(m, k, device="cuda"), torch.randn(k, n, device="cuda")
    with forced(F32TC=1):
        for sa, sb in ((1e-42, 1e20), (1e-38, 1.0), (1e-20, 1e-20), (1e37, 1e-37), (1e33, 1.0), (1e12, 1e13)):
            x, y = a * sa, b * sb
            want = product(x, y, 0, 0)
            got = matmul(x, y, 0, 0).double()
            # eight chains of k / 8 fused multiply-adds where the scaled range is left; results below 2^-126 are rounded to 2^-149
            assert (got - want).norm() <= (k / 8 + 3) * 2.0 ** -24 * product(x.abs(), y.abs(), 0, 0).norm() + (m * n) ** 0.5 * 2.0 ** -149, (sa, sb)
        a[3, 5], a[7, 1], b[9, 11], a[20, 9], a[50] = float("inf"), float("nan"), -float("inf"), 0.0, 3e38
        b[:, 60] = 1.0
        got, want = matmul(a, b, 0, 0), product(a, b, 0, 0).float()
        rows = torch.tensor([i for i in range(m) if i != 50], device="cuda")          # sums of 3e38: finite or not by their order
        assert torch.equal(torch.isnan(got[rows]), torch.isnan(want[rows])) and torch.equal(torch.isinf(got[rows]), torch.isinf(want[rows]))
        assert not torch.isfinite(got[50, 60])


# Everything out of the scaled range, and single infinities and NaN, with several tiles to a CTA, tiles split over clusters, pairs,
# and a K whose recomputation takes longer than the ring's waits last: equal to float64 but for rounding wherever that is finite
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("pair,bn,splits,m,k,n", [(0, 128, 8, 130, 1000, 200), (0, 32, 1, 2500, 40, 1027), (0, 96, 1, 2561, 33, 1537), (1, 256, 1, 5000, 40, 4099), (1, 192, 1, 300, 513, 260),
                                                  (0, 128, 8, 200, 1 << 16, 129), (1, 256, 1, 5200, 1 << 13, 1030)])
def test_f32_tensor_core_matmul_beyond_the_scaled_range(m, k, n, pair, bn, splits, ta, tb):
    a, b = torch.randn(*((k, m) if ta else (m, k)), device="cuda"), torch.randn(*((n, k) if tb else (k, n)), device="cuda")
    av, bv = a.t() if ta else a, b.t() if tb else b                                   # as M x K and K x N

    def run():
        with forced(F32TC=1, F32TC_PAIR=pair, F32TC_BN=bn, F32TC_SPLITS=splits):
            c = matmul(a, b, ta, tb).double()
        assert C.lib.b200jt_device_status() == 0
        return c, av.double() @ bv.double(), (av.double().abs() @ bv.double().abs())

    a *= 1e33                                                                          # all operands of one side beyond 2^104
    c, want, size = run()
    # parts of at most 256 of k by fused multiply-adds, added up one after the other; where K is split, up to eight more additions
    assert (c - want).norm() <= (256 / 8 + k / 256 + 8) * 2.0 ** -24 * size.norm()
    a /= 1e33
    av[m // 2, k // 3], bv[k // 2, n - 1], bv[k // 5, 0] = float("inf"), float("nan"), -float("inf")
    c, want, size = run()
    assert torch.equal(torch.isnan(c), torch.isnan(want)) and torch.equal(torch.isinf(c), torch.isinf(want))
    assert torch.equal(c[torch.isinf(c)], want[torch.isinf(want)])
    ok = torch.isfinite(want)
    assert (c[ok] - want[ok]).norm() <= (4 + k / 128) * 2.0 ** -23 * size[ok].norm()
    a.fill_(float("nan"))
    assert bool(torch.isnan(run()[0]).all())


def test_f32_matmul_without_scratch_stays_on_the_fma_pipe():
    a, b = torch.randn(600, 300, device="cuda"), torch.randn(300, 700, device="cuda")
    with forced(F32TC=0):
        want = matmul(a, b, 0, 0, scratch=False)
    with forced(F32TC=1):
        assert torch.equal(matmul(a, b, 0, 0, scratch=False), want)


def test_f32_tile_switches_do_not_outlast_or_precede_a_plan():
    """Switches of the tiles without that of the path: a thread that plans a size under them goes as one that does not."""
    import threading
    a, b, seen = torch.randn(500, 777, device="cuda"), torch.randn(777, 1000, device="cuda"), []

    def run():                                                                         # each thread plans for itself
        for _ in range(2):
            with forced(F32TC_SPLITS=1, F32TC_PAIR=0) if len(seen) == 2 else forced():
                seen.append(matmul(a, b, 0, 0))
    for _ in range(2):
        t = threading.Thread(target=run)
        t.start()
        t.join()
    assert len(seen) == 4 and all(torch.equal(seen[0], s) for s in seen[1:])


# ---- bfloat16 products whose last round alone is split (csrc/gemm_tcgen05.cu)
@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("pair,mt,bn,splits,m,k,n", [(0, 1, 64, 2, 1300, 300, 1000), (0, 1, 32, 3, 1283, 200, 500), (1, 1, 64, 4, 2570, 260, 600),
                                                     (1, 2, 32, 2, 5000, 136, 300)])
def test_bf16_matmul_split_last_round(pair, mt, bn, splits, m, k, n, ta, tb):
    a, b = torch.randn(*((k, m) if ta else (m, k)), device="cuda").bfloat16(), torch.randn(*((n, k) if tb else (k, n)), device="cuda").bfloat16()
    with forced(GEMM_PAIR=pair, GEMM_MT=mt, GEMM_BN=bn, GEMM_SPLITS=splits):
        c = matmul(a, b, ta, tb)
    want = product(a, b, ta, tb)
    assert (c.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()             # one rounding to bfloat16 of a float32 sum
    assert C.lib.b200jt_device_status() == 0


# ---- kernels that start while the pass before them drains: one after the other on one scratch buffer, with other inputs each time, give
# what each gives alone; also from a graph whose inputs change
def early_product(dtype, m, k, n, ta, tb):
    a, b = torch.randn(*((k, m) if ta else (m, k)), device="cuda").to(dtype), torch.randn(*((n, k) if tb else (k, n)), device="cuda").to(dtype)
    c = torch.empty(m, n, dtype=dtype, device="cuda")
    args = (C.desc(a), C.desc(b), C.desc(c), ta, tb)
    return [a, b], [c], int(C.lib.b200jt_matmul_workspace(*args)), lambda p, size: C.call("b200jt_matmul", *args, p, size)


def early_conv(kind, last):
    n, ci, co, side = 8, 64, 128, 28
    shape = lambda c: (n, side, side, c) if last else (n, c, side, side)
    x, y, w = torch.randn(shape(ci), device="cuda").bfloat16(), torch.randn(shape(co), device="cuda").bfloat16(), torch.randn(co, ci, 3, 3, device="cuda").bfloat16()
    fmt = (b"acdb", b"oihw", b"acdb") if last else (b"abcd", b"oihw", b"abcd")
    args = (C.desc(x), C.desc(w), C.desc(y), 1, 1, 1, 1, 1, 1, *fmt)
    if kind == "forward":
        stats = torch.empty(2 * co, device="cuda")
        return [x, w], [y, stats], int(C.lib.b200jt_conv2d_formats_workspace(*args)), lambda p, size: C.call("b200jt_conv2d_formats", *args, stats.data_ptr(), p, size)
    args = (C.desc(x), C.desc(y), C.desc(w), 1, 1, 1, 1, 1, 1, *fmt)
    return [x, y], [w], int(C.lib.b200jt_conv2d_backward_w_formats_workspace(*args)), lambda p, size: C.call("b200jt_conv2d_backward_w_formats", *args, p, size)


@pytest.mark.parametrize("make,args", [(early_product, (torch.float32, 500, 777, 1000, 0, 0)), (early_product, (torch.float32, 500, 777, 1000, 1, 1)),
                                       (early_product, (torch.bfloat16, 500, 777, 1000, 0, 0)), (early_conv, ("forward", 0)), (early_conv, ("forward", 1)),
                                       (early_conv, ("weights", 0)), (early_conv, ("weights", 1))])
def test_early_starts(make, args):
    calls = [make(*args) for _ in range(5)]
    size = calls[0][2]
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    run = lambda i: calls[i][3](ctypes.c_void_p(ws.data_ptr()), size)

    def alone():
        out = []
        for i in range(len(calls)):
            ws.fill_(0xff)                                                             # NaN, had anything read it too early
            torch.cuda.synchronize()
            run(i)
            torch.cuda.synchronize()
            out.append([t.clone() for t in calls[i][1]])
        return out

    def same(want):
        for i, w in enumerate(want):
            assert torch.equal(calls[i][1][0], w[0])
            for t, s in zip(calls[i][1][1:], w[1:]):                                   # channel sums: added up in the order of arrival
                assert (t - s).norm() <= 1e-5 * s.norm()
    want = alone()
    for _ in range(8):
        for i in range(len(calls)):
            run(i)
    same(want)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for i in range(len(calls)):
            run(i)
    for c in calls:
        for t in c[0]:
            t.copy_(torch.randn(t.shape, device="cuda"))
    want = alone()
    g.replay()
    g.replay()
    same(want)


# ---- few bins (csrc/reindex_reduce.cu): whole, part and no batches of a thread's two vectors
@pytest.mark.parametrize("op", ["add", "maximum"])
@pytest.mark.parametrize("dtype,idx", [(torch.float32, torch.int32), (torch.int32, torch.int32), (torch.float64, torch.int64)])
@pytest.mark.parametrize("n", [1 << 16, 148 * 8192, 148 * 8192 + 1, 148 * 16384 - 3, 148 * 24576 + 4099])
def test_few_bins(n, dtype, idx, op):
    import jittor_b200 as jt
    bins = 997
    v = torch.randint(-50, 50, (n,), device="cuda").to(dtype)                          # whole numbers: sums are exact in every order
    i = torch.randint(-2, bins + 2, (n,), device="cuda").to(idx)
    got = jt.array(v).reindex_reduce(op, [bins], ["@e0(i0)"], extras=[jt.array(i)]).torch()
    ok = (i >= 0) & (i < bins)
    if op == "add":
        want = torch.zeros(bins, device="cuda", dtype=torch.float64).index_add_(0, i[ok].long(), v[ok].double())
    else:
        want = torch.full((bins,), -1e9, device="cuda", dtype=torch.float64).scatter_reduce_(0, i[ok].long(), v[ok].double(), "amax")
    assert torch.equal(got.double(), want)


# skewed indices: bins above 1 % of a CTA's sample are summed in registers. Enough elements for that path, a ragged tail, indices that
# name no bin: negative ones, and 64-bit ones whose lower half is a hot bin's number
@pytest.mark.parametrize("idx", [torch.int32, torch.int64])
@pytest.mark.parametrize("hot", [1, 3, 6])
def test_few_bins_hot(hot, idx):
    import jittor_b200 as jt
    n, bins = 6_000_003, 997
    v = torch.randint(-9, 10, (n,), device="cuda").float()                             # whole numbers, sums below 2^24: exact in every order
    i = torch.randint(-3, bins + 3, (n,), device="cuda")
    spot = torch.randint(0, 2 * hot, (n,), device="cuda")
    i = torch.where(spot < hot, 7 + 150 * spot, i)
    if idx == torch.int64:
        i = torch.where(torch.rand(n, device="cuda") < 0.1, i + (1 << 32), i)
    got = jt.array(v).reindex_reduce("add", [bins], ["@e0(i0)"], extras=[jt.array(i.to(idx))]).torch()
    ok = (i >= 0) & (i < bins)
    assert torch.equal(got.double(), torch.zeros(bins, device="cuda", dtype=torch.float64).index_add_(0, i[ok], v[ok].double()))


# the fold behind the grid barrier: part of 32 bins, more bins than one pass of the grid takes, fewer CTAs; also from a graph
@pytest.mark.parametrize("reserve", [0, 64])
@pytest.mark.parametrize("dtype,bins", [(torch.float32, 1), (torch.float32, 33), (torch.int32, 4737), (torch.float32, 20011), (torch.float64, 9500)])
def test_few_bins_fold(dtype, bins, reserve):
    n = 300007
    v, i = torch.randint(-50, 50, (n,), device="cuda").to(dtype), torch.randint(0, bins, (n,), device="cuda", dtype=torch.int32)
    want = torch.zeros(bins, device="cuda", dtype=torch.float64).index_add_(0, i.long(), v.double())
    out = torch.empty(bins, dtype=dtype, device="cuda")
    idx, none = C.strings(["@e0(i0)"]), C.strings([])
    args = [C.desc(v), C.desc(out), b"add", idx, 1, none, 0, C.descs([i]), 1]
    ws = torch.empty(int(C.lib.b200jt_reindex_reduce_workspace(*args)), dtype=torch.uint8, device="cuda")
    run = lambda: C.call("b200jt_reindex_reduce", *args, ctypes.c_void_p(ws.data_ptr()), ws.numel())
    C.check(C.lib.b200jt_set_sm_reserve(reserve), "set_sm_reserve")
    try:
        run()
        assert torch.equal(out.double(), want)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            run()
        v.neg_()
        g.replay()
        g.replay()
        assert torch.equal(out.double(), -want)
    finally:
        C.lib.b200jt_set_sm_reserve(0)


# ---- softmax backward: rows in registers with the next one on its way, and rows of up to 16384 columns
@pytest.mark.parametrize("log", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(7, 127), (6, 129), (5, 511), (4, 2047), (3, 2049), (3, 4097), (2, 8191), (5, 8), (9500, 40), (2369, 2048), (4740, 1001), (3, 8192), (3, 8193), (150, 8200), (2, 12001), (2400, 16384), (2, 16383), (2, 16400)])
def test_softmax_backward(rows, cols, dtype, log):
    x = torch.randn(rows, cols, device="cuda")
    y = (torch.log_softmax(x, 1) if log else torch.softmax(x, 1)).to(dtype)
    dy, dx = torch.randn(rows, cols, device="cuda").to(dtype), torch.full((rows, cols), float("nan"), device="cuda", dtype=dtype)
    C.call("b200jt_softmax_backward", C.desc(y), C.desc(dy), C.desc(dx), log)
    yd, dd = y.double(), dy.double()
    want = dd - yd.exp() * dd.sum(1, keepdim=True) if log else yd * (dd - (yd * dd).sum(1, keepdim=True))
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    assert (dx.double() - want).norm() <= tol * want.norm()


# ---- pooling forward: two rows of two outputs to a thread (csrc/pool.cu)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k,stride,pad", [(2, 2, 0), (3, 2, 1), (3, 2, 0), (3, 1, 1)])
@pytest.mark.parametrize("h,w", [(4, 8), (5, 16), (8, 12), (11, 9), (10, 32), (13, 20)])
def test_pool_forward(h, w, k, stride, pad, dtype):
    import jittor_b200 as jt
    from jittor_b200 import pool
    x = torch.randn(3, 5, h, w, device="cuda").to(dtype)
    got = pool.max_pool2d(jt.array(x), k, stride, pad).torch()
    assert torch.equal(got, torch.nn.functional.max_pool2d(x, k, stride, pad))
    got = pool.avg_pool2d(jt.array(x), k, stride, pad).torch()
    want = torch.nn.functional.avg_pool2d(x.double(), k, stride, pad)
    assert (got.double() - want).abs().max() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21) * want.abs().max()


# ---- ragged rows: a warp, or a CTA of 64 to 1024 threads, to the row (csrc/rownorm.cu, csrc/norm_bwd.cu)
def placed(rows, cols, dtype, offset):
    """A [rows, cols] tensor that starts `offset` elements into a guarded buffer, and a check that the guards are untouched."""
    buf = torch.full((rows * cols + 32,), 7.0, device="cuda", dtype=dtype)
    t = buf[offset:offset + rows * cols].view(rows, cols)

    def guarded():
        return bool((buf[:offset] == 7).all()) and bool((buf[offset + rows * cols:] == 7).all())
    return t, guarded


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("rows,cols", [(1, 1), (9, 33), (19, 256), (2500, 257), (8200, 259), (5, 512), (21, 515), (2377, 1001), (5, 1024), (7, 1027),
                                       (601, 2051), (5, 4099), (3, 8191), (3, 8193)])
def test_ragged_rows(rows, cols, offset, dtype):
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 1e-5
    v = torch.randn(rows, cols, device="cuda").to(dtype)
    w = torch.randn(rows, cols, device="cuda").to(dtype)
    x, _ = placed(rows, cols, dtype, offset)
    dy, _ = placed(rows, cols, dtype, offset)
    x.copy_(v)
    dy.copy_(w)
    d = x.double()

    def near(got, want):
        return (got.double() - want).norm() <= tol * want.norm() + 1e-30
    for log in (0, 1):
        y, kept = placed(rows, cols, dtype, offset)
        C.call("b200jt_softmax", C.desc(x), C.desc(y), log)
        assert near(y, torch.log_softmax(d, 1) if log else torch.softmax(d, 1)) and kept()
        dx, kept = placed(rows, cols, dtype, offset)
        C.call("b200jt_softmax_backward", C.desc(y), C.desc(dy), C.desc(dx), log)
        yd, g = y.double(), dy.double()
        assert near(dx, g - yd.exp() * g.sum(1, keepdim=True) if log else yd * (g - (yd * g).sum(1, keepdim=True))) and kept()
    if cols < 2:
        return
    gamma, beta = torch.randn(cols, device="cuda"), torch.randn(cols, device="cuda")
    y, kept = placed(rows, cols, dtype, offset)
    C.call("b200jt_layer_norm", C.desc(x), C.desc(gamma), C.desc(beta), C.desc(y), 1e-5)
    d.requires_grad_(True)
    gd, bd = gamma.double().requires_grad_(True), beta.double().requires_grad_(True)
    want = torch.nn.functional.layer_norm(d, (cols,), gd, bd, 1e-5)
    assert near(y, want.detach()) and kept()
    if cols > 8192:
        return
    for pointer in (gamma, None):
        params = torch.full((2 * cols,), float("nan"), device="cuda")
        dx, kept = placed(rows, cols, dtype, offset)
        want = torch.nn.functional.layer_norm(d, (cols,), gd if pointer is not None else None, bd if pointer is not None else None, 1e-5)
        wx = torch.autograd.grad(want, d, dy.double())[0]
        n, p, ws = C.workspace("b200jt_layer_norm_backward_workspace", C.desc(x), 1)
        C.call("b200jt_layer_norm_backward", C.desc(x), C.desc(gamma) if pointer is not None else None, C.desc(dy), C.desc(dx), params.data_ptr(), 1e-5, p, n)
        xh = torch.nn.functional.layer_norm(d.detach(), (cols,), None, None, 1e-5)
        # two columns: the gradient is what is left of a cancellation, and E[x^2] - E[x]^2 loses digits with it
        assert (dx.double() - wx).norm() <= (tol if cols > 8 else 10 * tol) * (wx.norm() + 1e-2 * dy.double().norm()) and kept()
        assert near(params[:cols], (xh * dy.double()).sum(0)) and near(params[cols:], dy.double().sum(0))


# ---- BatchNorm's gradient in one launch (csrc/norm_bwd.cu): planes that do not divide the cluster, single elements, what shared
# memory just holds and what it does not; against float64, and the rounded forms against the two kernels
@pytest.mark.parametrize("form", [0, 1, 3, 5])
@pytest.mark.parametrize("xt,dt", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("shape", [(1, 2, 3, 3), (3, 5, 7, 7), (13, 3, 8, 8), (64, 128, 28, 28), (9, 40, 33, 31), (256, 512, 7, 7), (8, 2, 112, 128), (8, 2, 112, 136), (2, 1, 200, 200)])
def test_batch_norm_backward_in_one_launch(shape, xt, dt, form):
    cn, count = shape[1], shape[0] * shape[2] * shape[3]
    x, dy = (torch.randn(shape, device="cuda") + 0.3).to(xt), torch.randn(shape, device="cuda").to(dt)
    gamma, beta = torch.rand(cn, device="cuda") + 0.5, torch.randn(cn, device="cuda") * 0.1
    xd, per = x.double(), lambda t: t.double()[None, :, None, None]
    stats = torch.cat([xd.sum((0, 2, 3)), (xd * xd).sum((0, 2, 3))]).float()
    mean = per(stats[:cn].double() / count)
    rstd = (per(stats[cn:].double() / count) - mean ** 2 + 1e-5).rsqrt()
    xh = (xd - mean) * rstd
    act = xh * per(gamma) + per(beta)
    dy[act.abs() < 1e-4] = 0                               # within rounding of the ReLU's edge: either side of it is right
    dd = dy.double()
    head = (C.desc(x), C.desc(dy), stats.data_ptr(), float(count), gamma.data_ptr(), beta.data_ptr(), 1e-5, form)
    sums, dx = torch.full((4 * cn,), float("nan"), device="cuda"), torch.full(shape, float("nan"), device="cuda", dtype=xt)
    C.call("b200jt_bn_backward", *head, sums.data_ptr(), C.desc(dx))
    if form > 1:                                           # 16-bit steps: another order of the sums may turn one of them
        s2, d2 = torch.empty_like(sums), torch.empty_like(dx)
        C.call("b200jt_bn_backward_sums", *head, s2.data_ptr())
        C.call("b200jt_bn_backward_dx", *head, s2.data_ptr(), C.desc(d2))
        assert (sums - s2)[: 3 * cn].norm() <= 2.0 ** -7 * s2[: 3 * cn].norm() + 1e-5 * count ** 0.5 and (dx.double() - d2.double()).norm() <= 2.0 ** -7 * d2.double().norm()
        return
    d = torch.where(act > 0, dd, 0.0) if form else dd
    s0, s1 = d.sum((0, 2, 3)), (d * xh).sum((0, 2, 3))
    want = per(gamma) * rstd * (d - (per(s0) + xh * per(s1)) / count)
    assert (sums[:cn].double() - s0).norm() <= 1e-5 * count ** 0.5 * cn ** 0.5 and (sums[cn:2 * cn].double() - s1).norm() <= 1e-5 * count ** 0.5 * cn ** 0.5
    assert (dx.double() - want).norm() <= (2.0 ** -8 if xt == torch.bfloat16 else 1e-4) * want.norm() + 1e-6


@pytest.mark.parametrize("xt,dt", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("form", [2, 3, 4, 5])
@pytest.mark.parametrize("shape", [(3, 5, 7, 7), (13, 3, 8, 8), (64, 128, 28, 28), (256, 512, 7, 7), (2, 1, 200, 200)])
def test_batch_norm_backward_rounded_steps(shape, form, xt, dt):
    """The forms that round as a 16-bit graph does, step by step in torch: 2 and 3 with a float32 activation, 4 and 5 with every step to
    bfloat16, odd ones with a ReLU."""
    n, cn, hw = shape[0], shape[1], shape[2] * shape[3]
    count = float(n * hw)
    x, dy = (torch.randn(shape, device="cuda") + 0.3).to(xt), torch.randn(shape, device="cuda").to(dt)
    gamma, beta = torch.rand(cn, device="cuda") + 0.5, torch.randn(cn, device="cuda") * 0.1
    bf = lambda t: t.bfloat16().float()
    at = bf if form >= 4 else lambda t: t                                              # steps that only the second pair rounds
    per = lambda t: t[None, :, None, None]
    total = lambda t: t.double().sum((0, 2, 3)).float()
    xf, df, rc = x.float(), dy.float(), torch.tensor(1.0 / count, device="cuda")
    stats = torch.cat([total(xf), total(xf * xf)])
    mean, square = bf(stats[:cn] * rc), total(bf(xf * xf)) * rc
    sd = bf(bf(bf(bf(square) - bf(mean * mean)).clamp(min=0) + 1e-5).sqrt())
    w = at(gamma / sd)
    b = at(beta - at(mean * w))
    u = torch.where(at(xf * per(w)) + per(b) > 0, df, 0.0) if form % 2 else df
    s0, s1 = at(total(u)), at(total(at(xf * u)))
    dw = at(s1 + at(mean * -s0))
    dvar = bf(bf(at(-dw * gamma) / bf(sd * sd)) / bf(sd * 2))
    t = bf(mean * -dvar)
    p, q = bf(dvar * rc), bf(bf(bf(bf(w * -s0) + t) + t) * rc)
    step = bf(xf * per(p))
    want = bf(bf(bf(per(w) * u) + step) + step) + per(q)
    sums, dx = torch.full((4 * cn,), float("nan"), device="cuda"), torch.full(shape, float("nan"), device="cuda", dtype=xt)
    C.call("b200jt_bn_backward", C.desc(x), C.desc(dy), stats.data_ptr(), count, gamma.data_ptr(), beta.data_ptr(), 1e-5, form, sums.data_ptr(), C.desc(dx))
    # another order of the sums may turn a rounding of a channel's number, 2^-8 of it, and with it the channel's elements
    near = lambda got, ref, floor: (got.double() - ref.double()).norm() <= 2.0 ** -7 * ref.double().norm() + floor
    assert near(sums[:cn], s0, 1e-5 * count ** 0.5) and near(sums[2 * cn:3 * cn], square, 0)
    assert near(sums[3 * cn:], dw, 2.0 ** -7 * float((mean * s0).norm()) + 1e-5 * count ** 0.5)
    assert near(dx, want, 0)
