"""The packed path of the quantisers at the edges of its range: quotients around half integers, below -512 and above 512, of units whose
min_int is around -255 and 255, by rows and by a prompt's heads, against torch in the reference's arithmetic."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mean", [0.0, 12.4, 12.7, 12.8, -12.7, -12.75, -12.9, 25.6, 30.0, 400.0])
@pytest.mark.parametrize("rel", [0.05, 0.004])
@pytest.mark.parametrize("mode", ["ChannelQuant", "TokenQuant", "VectorQuant"])
def test_edges_of_the_packed_range(mean, rel, mode):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops
    if mean / rel > 65000:
        pytest.skip("quotients beyond fp16")
    m = ops.MODES[mode]
    g = torch.Generator(device="cuda").manual_seed(int(mean * 10) + 7)
    x = (torch.rand(128, 2, 3, 128, device="cuda", generator=g) + mean).half()
    x[::16] = mean                                             # (ties at the units' ends)
    x[:, :, 1] *= 0.01
    u = x.view(2, 64, 2, 3, 128) if mode == "ChannelQuant" else x.view(128, 1, 2, 3, 128)
    dims = {"ChannelQuant": (1,), "TokenQuant": (1, 3, 4), "VectorQuant": (1, 4)}[mode]
    step = ((u.amax(dims, keepdim=True) - u.amin(dims, keepdim=True)).float() * torch.tensor(rel, dtype=torch.float32, device="cuda")).half()
    low = (u.amin(dims, keepdim=True) / step).round()
    want = ((u / step).round() - low)                          # fp16 throughout, as the reference's tensors are
    ok = (want >= 0) & (want <= 255)
    n = ops.qspec(m, False, 2, 3, 128, 64).units(128, 2, 3, 128)
    mi, sc = torch.empty(n, dtype=torch.int16, device="cuda"), torch.empty(n, dtype=torch.float16, device="cuda")
    hist = torch.zeros(256, dtype=torch.int64, device="cuda")
    rows, _, _, _, _ = ops.quantize(x, m, 64, rel, False, min_dtype=torch.int16, hist=hist)
    heads = ops.quantize_heads(x.permute(1, 2, 0, 3).contiguous(), 128, None, None, m, 64, rel, False, mi, sc, None, ops.new_status(x.device))
    assert torch.equal(rows, heads) and torch.equal(hist, torch.bincount(rows.view(-1), minlength=256))
    assert torch.equal(rows.view(u.shape)[ok], want[ok].to(torch.uint8)) and float(ok.float().mean()) > 0.9
