"""bf16 tensor-core kernels at channel counts, extents, pitches and alignments that do not fit their tiles, against float64."""
import pytest
import torch

import jittor_b200 as jt
from jittor_b200 import _capi as C, nn

pytestmark = pytest.mark.gpu


def near(got, want):
    """One rounding to bf16 of sums accumulated in float32."""
    want = want.double()
    assert not got.isnan().any()
    assert (got.double() - want).abs().max() <= 2 ** -8 * want.abs().max() + 1e-30
    assert (got.double() - want).norm() <= 2 ** -8 * want.norm() + 1e-30


# channels below and across the 64-channel blocks, not multiples of 8; outputs smaller than a patch; 1 x 1 to 7 x 7 filters
@pytest.mark.parametrize("bn,pair", [(None, None), (64, 0), (64, 1), (128, 1), (256, 1)])
@pytest.mark.parametrize("n,ci,h,w,co,k,s,p,d", [
    (3, 8, 7, 7, 27, 3, 1, 1, 1), (2, 17, 9, 14, 16, 3, 1, 1, 1), (1, 63, 28, 28, 65, 1, 1, 0, 1), (2, 65, 16, 24, 130, 3, 2, 1, 1),
    (5, 33, 4, 5, 1, 2, 1, 1, 1), (2, 16, 56, 56, 112, 1, 2, 0, 1), (9, 129, 13, 8, 71, 5, 3, 2, 1), (1, 11, 40, 40, 300, 7, 4, 3, 2)])
def test_convolution_and_weight_gradient(n, ci, h, w, co, k, s, p, d, bn, pair, monkeypatch):
    if bn:
        monkeypatch.setenv("B200JT_CONV_BN", str(bn))
        monkeypatch.setenv("B200JT_CONV_PAIR", str(pair))
    x = torch.randn(n, ci, h, w, device="cuda").bfloat16()
    wt = (torch.randn(co, ci, k, k, device="cuda") * 0.1).bfloat16()
    wd = wt.double().requires_grad_()
    want = torch.nn.functional.conv2d(x.double(), wd, None, s, p, d)
    y = torch.full(list(want.shape), float("nan"), device="cuda").bfloat16()
    geo = (s, s, p, p, d, d)
    args = (C.desc(x), C.desc(wt), C.desc(y), *geo, 1)
    size, ptr, ws = C.workspace("b200jt_conv2d_workspace", *args)
    assert size > 0, "case does not reach the tensor-core kernel"
    stats = torch.full((2 * co,), 7.0, device="cuda")
    C.call("b200jt_conv2d", *args, stats.data_ptr(), ptr, size)
    near(y, want)
    yd = y.double()
    assert torch.allclose(stats[:co].double(), yd.sum((0, 2, 3)), rtol=0, atol=1e-4 * float(yd.abs().sum((0, 2, 3)).max()) + 1e-6)
    assert torch.allclose(stats[co:].double(), (yd * yd).sum((0, 2, 3)), rtol=1e-4, atol=1e-6)
    dy = torch.randn(*want.shape, device="cuda").bfloat16()
    want.backward(dy.double())
    dw = torch.full(list(wt.shape), float("nan"), device="cuda").bfloat16()
    dy = torch.cat([dy.flatten()[:1], dy.flatten()])[1:].view_as(dy)               # 2-byte aligned
    args = (C.desc(x), C.desc(dy), C.desc(dw), *geo)
    size, ptr, ws = C.workspace("b200jt_conv2d_backward_w_workspace", *args)
    C.call("b200jt_conv2d_backward_w_tc", *args, ptr, size)
    near(dw, wd.grad)
    assert C.lib.b200jt_device_status() == 0


# (M, N, K): extents around the tiles (128 / 256 / 512 rows, 32 .. 256 columns, 64 of K), pitches that are not multiples of 8,
# products below one tile, K long enough to be split
SIZES = [(64, 64, 64), (16, 4096, 512), (129, 33, 77), (513, 257, 130), (300, 10, 1000), (128, 256, 4096), (1031, 519, 321),
         (2, 1000, 2048), (520, 601, 40), (4096, 64, 96)]
VARIANTS = [{}, {"PAIR": 0, "BN": 32}, {"PAIR": 0, "BN": 224, "SPLITS": 3}, {"PAIR": 1, "MT": 1, "BN": 96}, {"PAIR": 1, "MT": 1, "BN": 256},
            {"PAIR": 1, "MT": 2, "BN": 160, "SPLITS": 2}, {"PAIR": 1, "MT": 2, "BN": 256}]


@pytest.mark.parametrize("variant", VARIANTS, ids=lambda v: "-".join(f"{k}{x}" for k, x in v.items()) or "chosen")
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_matmul(ta, tb, variant, monkeypatch):
    for k, v in variant.items():
        monkeypatch.setenv("B200JT_GEMM_" + k, str(v))
    for m, n, k in SIZES:
        a = torch.randn(*((k, m) if ta else (m, k)), device="cuda").bfloat16()
        b = torch.randn(*((n, k) if tb else (k, n)), device="cuda").bfloat16()
        c = torch.full((m, n), float("nan"), device="cuda").bfloat16()
        args = (C.desc(a), C.desc(b), C.desc(c), ta, tb)
        size, ptr, ws = C.workspace("b200jt_matmul_workspace", *args)
        want = (a.double().t() if ta else a.double()) @ (b.double().t() if tb else b.double())
        C.call("b200jt_matmul", *args, ptr, size)
        near(c, want)
        if ta == 0 and n * m < 4096:                        # 2-byte aligned operand: the CUDA-core kernel
            a1 = torch.randn(a.numel() + 1, device="cuda").bfloat16()[1:].view_as(a)
            C.call("b200jt_matmul", C.desc(a1), *args[1:], ptr, size)
            near(c, a1.double() @ (b.double().t() if tb else b.double()))
    assert C.lib.b200jt_device_status() == 0


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_batched_matmul(ta, tb, pair, monkeypatch):
    monkeypatch.setenv("B200JT_GEMM_PAIR", str(pair))
    for ba, bb, m, n, k in [(3, 3, 128, 64, 64), (1, 5, 136, 72, 200), (4, 1, 520, 264, 72)]:
        a = torch.randn(ba, *((k, m) if ta else (m, k)), device="cuda").bfloat16()
        b = torch.randn(bb, *((n, k) if tb else (k, n)), device="cuda").bfloat16()
        c = torch.full((max(ba, bb), m, n), float("nan"), device="cuda").bfloat16()
        C.call("b200jt_batched_matmul", C.desc(a), C.desc(b), C.desc(c), ta, tb)
        near(c, (a.double().transpose(1, 2) if ta else a.double()) @ (b.double().transpose(1, 2) if tb else b.double()))
    assert C.lib.b200jt_device_status() == 0


@pytest.mark.parametrize("n,ci,h,w,co,k,s,p,d", [(3, 5, 27, 33, 8, 3, 2, 1, 1), (2, 70, 16, 16, 9, 1, 2, 0, 1), (4, 16, 29, 24, 24, 5, 3, 2, 1),
                                                 (2, 8, 40, 23, 64, 2, 4, 0, 1), (1, 24, 21, 21, 16, 3, 2, 2, 2), (2, 9, 9, 9, 4, 3, 2, 1, 1)])
def test_strided_input_gradient(n, ci, h, w, co, k, s, p, d):
    x, wt = torch.randn(n, ci, h, w, device="cuda").bfloat16(), (torch.randn(co, ci, k, k, device="cuda") * 0.1).bfloat16()
    vx = jt.array(x)
    y = nn.conv2d(vx, jt.array(wt), None, s, p, d)
    dy = torch.randn(*y.shape, device="cuda").bfloat16()
    got = jt.grad((y * jt.array(dy)).sum(), vx).torch()
    xd = x.double().requires_grad_()
    torch.nn.functional.conv2d(xd, wt.double(), None, s, p, d).backward(dy.double())
    near(got, xd.grad)


@pytest.mark.parametrize("ci,h,w,co,k,s,p", [(96, 20, 20, 64, 3, 1, 1), (200, 9, 13, 300, 3, 1, 1), (64, 28, 28, 128, 5, 2, 2), (320, 7, 7, 96, 1, 1, 0)])
def test_an_image_gives_the_same_bits_at_every_place_of_a_batch(ci, h, w, co, k, s, p):
    x = torch.randn(1, ci, h, w, device="cuda").bfloat16().expand(37, -1, -1, -1).contiguous()
    wt = jt.array((torch.randn(co, ci, k, k, device="cuda") * 0.1).bfloat16())
    y = nn.conv2d(jt.array(x), wt, None, s, p)
    assert all(torch.equal(y.torch()[0], image) for image in y.torch())


# filters that reach as far as an im2col map allows: corners at -128 and 127, shifts up to 255
@pytest.mark.parametrize("n,ci,h,w,co,k,p,d", [(1, 64, 80, 72, 64, 3, 64, 64), (2, 8, 140, 131, 16, 3, 127, 127), (1, 16, 20, 9, 24, 2, 128, 255),
                                               (1, 24, 150, 160, 8, 2, 0, 128), (1, 8, 30, 30, 8, 1, 127, 1)])
def test_convolution_of_wide_reach(n, ci, h, w, co, k, p, d, monkeypatch):
    test_convolution_and_weight_gradient(n, ci, h, w, co, k, 1, p, d, None, None, monkeypatch)


def test_input_gradient_with_float32_weights():
    """The weights are cast for the launch; the scratch memory allocated after that is not theirs."""
    from jittor_b200 import executor
    dy, w = torch.randn(2, 256, 14, 14, device="cuda").bfloat16(), torch.randn(256, 256, 3, 3, device="cuda") * 0.02
    xd = torch.zeros(2, 256, 28, 28, device="cuda", dtype=torch.float64, requires_grad=True)
    torch.nn.functional.conv2d(xd, w.bfloat16().double(), None, 2, 1).backward(dy.double())
    plan = executor.conv_dx_plan(jt.Var([2, 256, 28, 28], "bfloat16"), jt.array(dy), jt.array(w), (2, 2, 1, 1, 1, 1))
    C.recorder = rec = C.Recorder([p._data for p in plan.leaves])          # takes no pointer to memory that was given back
    try:
        got = plan.run()
    finally:
        C.recorder = None
    assert rec.ok
    near(got, xd.grad)


@pytest.mark.parametrize("shape", [(3, 5, 1, 300), (202, 7, 7, 7), (37, 3, 1, 1023), (9, 4, 16, 16), (600, 2, 1, 1), (300, 150, 2, 3)])
@pytest.mark.parametrize("op", ["mean", "add", "maximum"])
def test_reduction_over_short_rows(shape, op):
    x = torch.randn(*shape, device="cuda")
    y = torch.empty(1, shape[1], 1, 1, device="cuda")
    args = (C.desc(x), C.desc(y), op.encode(), 0b1101)
    size, ptr, ws = C.workspace("b200jt_reduce_workspace", *args)
    C.call("b200jt_reduce", *args, ptr, size)
    xd = x.double()
    want = xd.amax((0, 2, 3)) if op == "maximum" else xd.mean((0, 2, 3)) if op == "mean" else xd.sum((0, 2, 3))
    assert torch.allclose(y.flatten().double(), want, rtol=1e-5, atol=1e-5 * float(xd.abs().sum((0, 2, 3)).max() if op == "add" else 1))
