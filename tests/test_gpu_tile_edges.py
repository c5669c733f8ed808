"""Kernels at the sizes where their tiles, rings, splits and register rows begin and end, against float64 (or exactly)."""
import pytest
import torch

from jittor_b200 import _capi as C

pytestmark = pytest.mark.gpu


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
