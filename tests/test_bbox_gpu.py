"""Bounding box kernel against torch's column minimum and maximum: sizes around a group of eight points, a block and the
switch to two launches, unaligned starts, columns with NaN and infinities."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 4095, 4096, 32768, 32769, 200003, 1300001])
@pytest.mark.parametrize("skip", [0, 1])
@pytest.mark.parametrize("special", [None, "nan", "inf"])
def test_bounding_box(cuda_device, n, skip, special):
    from flash3dtransformer_b200.psh import psh_main
    g = torch.Generator(cuda_device).manual_seed(n + skip)
    c = ((torch.rand(n + skip, 3, generator=g, device=cuda_device) - 0.3) * 100).half()[skip:]
    if special == "nan":
        c[n // 2, 1] = float("nan")
    elif special == "inf":
        c[0, 0], c[n - 1, 2] = float("inf"), float("-inf")
    lo, hi = psh_main.bounding_box(c)
    ref = torch.aminmax(c, dim=0)
    assert torch.equal(lo.isnan(), ref.min.isnan()) and torch.equal(hi.isnan(), ref.max.isnan())
    assert torch.equal(lo.nan_to_num(0), ref.min.nan_to_num(0)) and torch.equal(hi.nan_to_num(0), ref.max.nan_to_num(0))
