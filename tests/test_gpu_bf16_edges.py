"""bf16 tensor-core kernels at channel counts, extents, pitches and alignments that do not fit their tiles, against float64."""
import pytest
import torch

from jittor_b200 import _capi as C

pytestmark = pytest.mark.gpu


def near(got, want):
    """One rounding to bf16 of sums accumulated in float32."""
    want = want.double()
    assert not got.isnan().any()
    assert (got.double() - want).abs().max() <= 2 ** -8 * want.abs().max() + 1e-30
    assert (got.double() - want).norm() <= 2 ** -8 * want.norm() + 1e-30


# channels below and across the 64-channel blocks, not multiples of 8; outputs smaller than a patch; 1 x 1 to 7 x 7 filters
@pytest.mark.parametrize("bn", [None, 64])
@pytest.mark.parametrize("n,ci,h,w,co,k,s,p,d", [
    (3, 8, 7, 7, 27, 3, 1, 1, 1), (2, 17, 9, 14, 16, 3, 1, 1, 1), (1, 63, 28, 28, 65, 1, 1, 0, 1), (2, 65, 16, 24, 130, 3, 2, 1, 1),
    (5, 33, 4, 5, 1, 2, 1, 1, 1), (2, 16, 56, 56, 112, 1, 2, 0, 1), (9, 129, 13, 8, 71, 5, 3, 2, 1), (1, 11, 40, 40, 300, 7, 4, 3, 2)])
def test_convolution_and_weight_gradient(n, ci, h, w, co, k, s, p, d, bn, monkeypatch):
    if bn:
        monkeypatch.setenv("B200JT_CONV_BN", str(bn))
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
    args = (C.desc(x), C.desc(dy), C.desc(dw), *geo)
    size, ptr, ws = C.workspace("b200jt_conv2d_backward_w_workspace", *args)
    C.call("b200jt_conv2d_backward_w_tc", *args, ptr, size)
    near(dw, wd.grad)
    assert C.lib.b200jt_device_status() == 0
