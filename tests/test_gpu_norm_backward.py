"""Gradient kernels of LayerNorm and training BatchNorm (csrc/norm_bwd.cu) and the one-element row kernels (csrc/rownorm.cu) at
the edges of their register tiles, against float64 and, for bfloat16 BatchNorm, against the meta-op graph they stand for."""
import numpy as np
import pytest
import torch

import jittor_b200 as jt
from jittor_b200 import nn
from jittor_b200.grad import backprop

pytestmark = pytest.mark.gpu


def near(got, want, tol):
    assert (got.double() - want.double()).norm() <= tol * want.double().norm() + 1e-12


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 7), (40, 255), (33, 256), (2000, 264), (7, 513), (100, 1001), (9, 1024), (5, 1025), (64, 2049),
                                       (300, 4096), (3, 4100), (2, 8191), (2, 8192)])
def test_layer_norm_and_softmax(rows, cols, dtype):
    x, dy = (torch.randn(rows, cols, device="cuda").to(dtype) for _ in range(2))
    g, b = 1 + 0.1 * torch.randn(cols, device="cuda"), torch.randn(cols, device="cuda")
    vx, vg, vb, vdy = jt.array(x), jt.array(g), jt.array(b), jt.array(dy)
    y = nn.layer_norm(vx, (cols,), vg, vb)
    dx, dg, db = jt.grad((y * vdy).sum(), [vx, vg, vb])
    jt.sync([y, dx, dg, db])
    xd, gd, bd = (t.double().requires_grad_() for t in (x, g, b))
    ref = torch.nn.functional.layer_norm(xd, (cols,), gd, bd)
    ref.backward(dy.double())
    tol = 1e-5 if dtype == torch.float32 else 6e-3
    if cols > 1:
        near(y.torch(), ref.detach(), tol)
        near(dx.torch(), xd.grad, tol)
        near(dg.torch(), gd.grad, 1e-5)
    near(db.torch(), bd.grad, 1e-5)
    only = jt.grad((nn.layer_norm(vx, (cols,), vg, vb) * vdy).sum(), vx)             # without the parameters' sums
    assert torch.equal(only.torch(), dx.torch())
    for log in (False, True):
        s = nn.softmax(vx, -1, log)
        ds = jt.grad((s * vdy).sum(), vx)
        jt.sync([s, ds])
        xs = x.double().requires_grad_()
        ref = torch.log_softmax(xs, -1) if log else torch.softmax(xs, -1)
        ref.backward(dy.double())
        near(s.torch(), ref.detach(), tol)
        if cols > 1 and dtype == torch.float32:
            near(ds.torch(), xs.grad, 2e-5)


@pytest.mark.parametrize("dtype,amp", [(torch.float32, 0), (torch.bfloat16, 0), (torch.bfloat16, 2)])
@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("n,c,h,w", [(2, 1, 3, 5), (2, 3, 5, 7), (33, 5, 7, 7), (4, 16, 16, 16), (64, 130, 4, 4), (3, 700, 9, 8)])
def test_batch_norm(n, c, h, w, relu, dtype, amp):
    with jt.flag_scope(amp_reg=amp):
        bn = nn.BatchNorm(c)
        bn.weight, bn.bias = jt.array(1 + 0.1 * torch.randn(c, device="cuda")), jt.array(0.3 * torch.randn(c, device="cuda"))
        vx = jt.array((torch.randn(n, c, h, w, device="cuda") + 0.2).to(dtype))
        y = nn.relu(bn(vx)) if relu else bn(vx)
        vdy = jt.array(torch.randn(n, c, h, w, device="cuda").to(torch.bfloat16 if y.dtype == "bfloat16" else torch.float32))
        targets = [vx, bn.weight, bn.bias]
        got = jt.grad((y * vdy).sum(), targets)
        jt.sync([y] + got)
        root = y._relay[1] if relu else y
        node = jt.Var(root.shape, root.dtype, root._op)                               # the graph itself, op by op
        want = backprop(jt.ternary(node > 0.0, node, 0.0) if relu else node, vdy, targets)
        for a, b in zip(got, want):
            if dtype == torch.float32:
                near(a.torch(), b.torch(), 1e-4)
            else:
                near(a.torch(), b.torch(), 4e-3 if amp == 0 else 1e-3)    # amp 2 rounds as the graph does: at most a flip here and there


@pytest.mark.parametrize("weight,bias", [(2.0, 0.5), (0.0, 1.0), (np.full(6, 2.0, np.float32), np.full(6, 0.5, np.float32)), (1.0, -3.0)])
@pytest.mark.parametrize("relu", [False, True])
def test_batch_norm_with_numbers_for_parameters(weight, bias, relu):
    x, dy = torch.randn(5, 6, 7, 9, device="cuda") + 0.2, torch.randn(5, 6, 7, 9, device="cuda")
    bn, vx = nn.BatchNorm(6), jt.array(x)
    bn.weight, bn.bias = weight, bias
    y = nn.relu(bn(vx)) if relu else bn(vx)
    dx = jt.grad((y * jt.array(dy)).sum(), vx)
    jt.sync([y, dx])
    xd = x.double().requires_grad_()
    w, b = (torch.as_tensor(p, device="cuda").double().expand(6) for p in (weight, bias))
    ref = torch.nn.functional.batch_norm(xd, None, None, w, b, True, eps=1e-5)
    ref = torch.relu(ref) if relu else ref
    ref.backward(dy.double())
    near(y.torch(), ref.detach(), 1e-5)
    near(dx.torch(), xd.grad, 1e-4)
    near(bn.running_mean.torch(), 0.1 * x.double().mean((0, 2, 3)), 1e-5)


@pytest.mark.parametrize("replaced", ["float64", "shape"])
def test_running_statistics_the_kernel_does_not_move(replaced):
    """Statistics of another dtype or shape than the kernel's float32 [C] move through the graph's."""
    x = torch.randn(5, 6, 7, 9, device="cuda") + 0.2
    want = 0.1 * x.double().mean((0, 2, 3))
    for _ in range(3):                                    # planned, then from what the first run left
        bn = nn.BatchNorm(6)
        if replaced == "float64":
            bn.running_mean, bn.running_var = jt.zeros((6,), "float64"), jt.ones((6,), "float64")
        else:
            bn.running_mean, bn.running_var = jt.zeros((1,)), jt.ones((1,))
        bn(jt.array(x)).sync()
        near(bn.running_mean.torch(), want, 1e-5)


def test_batch_norm_sums_over_more_than_2_31_elements_of_a_channel():
    from jittor_b200 import _capi as C
    n, h, w = 16, 32767, 32771                            # odd planes: one element per access, 2 * h * w > 2^31 of them for a CTA
    x = torch.ones(n, 1, h, w, device="cuda", dtype=torch.bfloat16)
    stats, sums = torch.zeros(2, device="cuda"), torch.empty(4, device="cuda")
    C.call("b200jt_bn_backward_sums", C.desc(x), C.desc(x), stats.data_ptr(), float(n * h * w), None, None, 1e-5, 0, sums.data_ptr())
    assert abs(sums[0].item() - n * h * w) <= 1e-6 * n * h * w          # each thread counts up to 2^23 ones: exact until the threads meet
    del x
    torch.cuda.empty_cache()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cols", [7, 255, 256, 1001, 1024, 4100, 8191, 8192, 16384, 32768, 40001])
def test_softmax_of_rows_that_are_masked_as_a_whole(cols, dtype):
    """Rows of the type's lowest value, as an additive mask leaves them, are rows of equal elements."""
    low = torch.finfo(dtype).min
    x = torch.full((4, cols), low, device="cuda", dtype=dtype)
    x[1, cols // 2] = 1.0
    x[2, 0], x[2, 1:] = -3e38, low
    x[3] = torch.linspace(-2e38, -1.9e38, cols, device="cuda").to(dtype)
    for log in (False, True):
        got = nn.softmax(jt.array(x), -1, log).torch().double()
        want = torch.log_softmax(x.double(), -1) if log else torch.softmax(x.double(), -1)
        assert torch.isfinite(got[:2]).all() and not got.isnan().any()
        tol = 1e-5 if dtype == torch.float32 else 2 ** -7
        if log:                                               # differences of huge numbers: what float32 holds of them
            assert torch.allclose(got[:1], want[:1], rtol=tol, atol=0)
        else:
            assert torch.allclose(got, want, rtol=tol, atol=1e-30)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cols", [8, 256, 1024, 4096, 8192, 16384])
@pytest.mark.parametrize("which", [(0,), (1,), (0, 1)])
def test_layer_norm_parameters_at_odd_addresses(cols, dtype, which):
    """Parameters that are views into a larger tensor, four bytes off, beside rows at 16-byte addresses."""
    x = torch.randn(5, cols, device="cuda").to(dtype)
    par = [1 + 0.1 * torch.randn(cols, device="cuda"), torch.randn(cols, device="cuda")]
    for i in which:
        par[i] = torch.cat([par[i][:1], par[i]])[1:]
        assert par[i].data_ptr() % 16
    y = nn.layer_norm(jt.array(x), (cols,), jt.array(par[0]), jt.array(par[1]))
    want = torch.nn.functional.layer_norm(x.double(), (cols,), par[0].double(), par[1].double())
    near(y.torch(), want, 1e-5 if dtype == torch.float32 else 6e-3)
