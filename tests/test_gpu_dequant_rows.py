"""Per-channel dequantisation of several tokens by a thread: around the size from which it is taken, lengths that are no multiple of its tokens, both widths of min_int."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,H,block", [(64, 8, 74, 64), (64, 8, 75, 64), (320, 8, 20, 64), (256, 5, 31, 128), (130, 9, 33, 2), (63, 16, 40, 3), (128, 40, 8, 64)])
@pytest.mark.parametrize("dtype", [torch.int8, torch.int16])
def test_values(T, B, H, block, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T + H)
    spec = ops.qspec(ops.MODE_CHANNEL, False, B, H, 128, block)
    n = spec.units(T, B, H, 128)
    codes = torch.randint(0, 256, (T, B, H, 128), dtype=torch.uint8, device="cuda", generator=g)
    mi = torch.randint(-128, 128, (n,), device="cuda", generator=g).to(dtype)
    if dtype == torch.int16:
        mi[::7] *= 200
    sc = (torch.rand(n, device="cuda", generator=g) + 0.01).half()
    u = (T // block, 1, B, H, 128)
    want = ((codes.view(T // block, block, B, H, 128).int() + mi.view(u).int()).half() * sc.view(u)).view(codes.shape)      # the sum in whole numbers
    assert torch.equal(ops.dequant(codes, mi, sc, spec), want)


# around 512 threads per SM, from where a thread takes several tokens
@pytest.mark.parametrize("T,B,H,block", [(64, 1, 74, 64), (64, 1, 75, 64), (65, 3, 33, 5), (128, 2, 19, 2)])
@pytest.mark.parametrize("dtype", [torch.int8, torch.int16])
def test_values_of_small_calls(T, B, H, block, dtype):
    test_values(T, B, H, block, dtype)
