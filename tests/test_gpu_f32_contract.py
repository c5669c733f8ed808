"""float32 contraction kernel (csrc/gemm_f32.cu) at the edges of its tiles, splits and residue classes, against float64."""
import pytest
import torch

import jittor_b200 as jt
from jittor_b200 import _capi as C, nn

pytestmark = pytest.mark.gpu


def near(got, want):
    want = want.double()
    assert (got.double() - want).norm() <= 1e-5 * want.norm() + 1e-30
    assert (got.double() - want).abs().max() <= 1e-4 * want.abs().max() + 1e-30


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (33, 1, 7), (15, 17, 16), (63, 65, 48), (128, 128, 50), (129, 130, 257), (16, 10, 2048),
                                   (500, 77, 333), (1030, 516, 64), (2, 3000, 5)])
def test_matmul(m, n, k, ta, tb):
    a = torch.randn(*((k, m) if ta else (m, k)), device="cuda")
    b = torch.randn(*((n, k) if tb else (k, n)), device="cuda")
    c = torch.empty(m, n, device="cuda")
    args = (C.desc(a), C.desc(b), C.desc(c), ta, tb)
    size, ptr, ws = C.workspace("b200jt_matmul_workspace", *args)
    want = (a.double().t() if ta else a.double()) @ (b.double().t() if tb else b.double())
    for p, s in ((ptr, size), (None, 0)):               # with the scratch it asks for, and without
        c.fill_(float("nan"))
        C.call("b200jt_matmul", *args, p, s)
        near(c, want)
    if k > 1:                                           # 4-byte aligned operands
        a1 = torch.randn(a.numel() + 1, device="cuda")[1:].view_as(a)
        C.call("b200jt_matmul", C.desc(a1), *args[1:], ptr, size)
        near(c, (a1.double().t() if ta else a1.double()) @ (b.double().t() if tb else b.double()))


@pytest.mark.parametrize("n,ci,h,w,co,k,s,p,d", [
    (1, 1, 1, 1, 1, 1, 1, 0, 1), (2, 3, 9, 8, 5, 3, 1, 1, 1), (4, 32, 32, 32, 64, 3, 1, 1, 1), (1, 64, 7, 7, 33, 3, 1, 2, 2),
    (3, 4, 10, 10, 6, 2, 4, 1, 1), (5, 7, 9, 11, 13, 3, 3, 2, 2), (8, 3, 63, 60, 37, 5, 2, 2, 1), (2, 5, 8, 8, 3, 1, 2, 0, 1),
    (16, 17, 13, 12, 130, 3, 2, 1, 1), (70, 3, 20, 20, 16, 3, 1, 1, 1)])
def test_conv_and_its_gradients(n, ci, h, w, co, k, s, p, d):
    x, wt = torch.randn(n, ci, h, w, device="cuda"), torch.randn(co, ci, k, k, device="cuda")
    want = torch.nn.functional.conv2d(x.double(), wt.double(), stride=s, padding=p, dilation=d)
    dy = torch.randn(want.shape, device="cuda")
    vx, vw = jt.array(x), jt.array(wt)
    y = nn.conv2d(vx, vw, None, s, p, d)
    dx, dw = jt.grad((y * jt.array(dy)).sum(), [vx, vw])
    jt.sync([y, dx, dw])
    near(y.torch(), want)
    near(dx.torch(), torch.nn.grad.conv2d_input(x.shape, wt.double(), dy.double(), stride=s, padding=p, dilation=d))
    near(dw.torch(), torch.nn.grad.conv2d_weight(x.double(), wt.shape, dy.double(), stride=s, padding=p, dilation=d))
    again = torch.empty_like(wt)                        # without scratch: fewer slices, the same sums
    C.call("b200jt_conv2d_backward_w", C.desc(x), C.desc(dy), C.desc(again), s, s, p, p, d, d)
    near(again, dw.torch())


def test_batched_matmul():
    a, b = torch.randn(7, 33, 50, device="cuda"), torch.randn(1, 50, 19, device="cuda")
    near(nn.bmm(jt.array(a), jt.array(b)).torch(), a.double() @ b.double())
