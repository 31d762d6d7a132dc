"""The sum over the unfused P.V's groups: below, at and beyond a round of eight rows per warp and of 64 per CTA."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 63, 64, 65, 128, 300])
@pytest.mark.parametrize("B,Hq", [(1, 1), (3, 5), (2, 32)])
def test_sum_of_groups(n, B, Hq):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops
    part = torch.randn(n, B, Hq, 128, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)).half()
    got = ops.pv_sum(part)
    want = part.double().sum(dim=0, keepdim=True)
    # half an ulp of fp16, and fp32 sums of n values of magnitude up to 5: n ulps of the sum of magnitudes at most
    bound = want.abs() * 2.0 ** -11 + part.double().abs().sum(dim=0, keepdim=True) * n * 2.0 ** -24 + 2.0 ** -25
    assert got.shape == want.shape and bool(((got.double() - want).abs() <= bound).all())
