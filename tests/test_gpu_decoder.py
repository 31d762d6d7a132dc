"""The decoder's pairs of warps over every split of the blocks: one block, fewer blocks than SMs, a ragged last round; known
and unknown largest block; a stream that does not start on 16 bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("is_k", [True, False])
@pytest.mark.parametrize("B,H,T", [(1, 1, 128), (1, 3, 256), (2, 10, 896), (1, 37, 1280), (3, 32, 1536)])
def test_blocks_over_pairs_of_warps(ops, is_k, B, H, T):
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, B, H, 128, device="cuda", generator=g).half()
    mode = ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN
    hist = torch.zeros(256, dtype=torch.int64, device="cuda")
    codes, mi, sc, spec, _ = ops.quantize(x, mode, 64, 0.05, False, min_dtype=torch.int16, hist=hist)
    book = ops.build_codebook(hist)
    bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
    bi, ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz, dtype=torch.uint8, device="cuda")
    for shift in (0, 5):
        enc = torch.empty(n + 16, dtype=torch.uint8, device="cuda")[shift:]
        total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
        size, largest = total.tolist()
        assert ops.read_status(st) == 0
        for bound in (0, largest):
            back, st = ops.decode(enc[:size], bi, ti, book, T, B, H, is_k, max_block=bound)
            assert ops.read_status(st) == 0 and torch.equal(back, codes)
            out = torch.empty(T, B, H, 128, dtype=torch.float16, device="cuda")
            st = ops.decode_values(ops.make_cache(enc, bi, ti, book, mi, sc, spec, size, bound), T, B, H, is_k, out)
            assert ops.read_status(st) == 0 and torch.equal(out.view(torch.int16), ops.dequant(codes, mi, sc, spec).view(torch.int16))
