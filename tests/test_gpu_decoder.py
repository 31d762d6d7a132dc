"""The decoder's pairs of warps over every split of the blocks: one block, fewer blocks than SMs, a ragged last round; known
and unknown largest block; a stream that does not start on 16 bytes."""
import numpy as np
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


@pytest.mark.parametrize("is_k", [True, False])
@pytest.mark.parametrize("B,H,T,leads", [(1, 1, 128, range(16)), (8, 40, 1024, (0, 3, 15))])
def test_streams_that_end_with_their_memory(ops, is_k, B, H, T, leads):
    """No byte behind the stream is asked for: the block whose 16-byte chunks pass the end comes by plain loads, be it the
    last one of the launch or, with blocks in another order, one that the pair goes on from."""
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, B, H, 128, device="cuda", generator=g).half()
    hist = torch.zeros(256, dtype=torch.int64, device="cuda")
    codes, mi, sc, spec, _ = ops.quantize(x, ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN, 64, 0.05, False, min_dtype=torch.int16, hist=hist)
    book = ops.build_codebook(hist)
    bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
    bi, ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz, dtype=torch.uint8, device="cuda")
    enc = torch.empty(n, dtype=torch.uint8, device="cuda")
    total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
    size, largest = total.tolist()
    assert ops.read_status(st) == 0
    values = ops.dequant(codes, mi, sc, spec)
    rec = bi.cpu().numpy().view(np.uint32).reshape(-1, 2)
    count = (rec[:, 1] & 0xffff).astype(np.int64)
    host = enc[:size].cpu().numpy()
    ends = set()
    for lead in leads:
        order = np.random.default_rng(lead).permutation(len(rec)) if lead % 2 else np.arange(len(rec))
        at = np.empty(len(rec), np.int64)
        at[order] = lead + np.concatenate(([0], np.cumsum(count[order])[:-1]))
        stream = np.full(lead + size, 0xff, np.uint8)
        for i in range(len(rec)):
            stream[at[i]:at[i] + count[i]] = host[rec[i, 0]:rec[i, 0] + count[i]]
        moved = rec.copy()
        moved[:, 0] = at
        dbi = torch.from_numpy(moved.view(np.uint8).reshape(-1)).cuda()
        whole = torch.full((lead + size + 64,), 0xff, dtype=torch.uint8, device="cuda")
        whole[:lead + size] = torch.from_numpy(stream).cuda()
        cut = whole[:lead + size]
        assert cut.data_ptr() % 16 == 0
        ends.add((lead + size) % 16)
        for bound in (0, largest):
            back, st = ops.decode(cut, dbi, ti, book, T, B, H, is_k, max_block=bound)
            assert ops.read_status(st) == 0 and torch.equal(back, codes)
            out = torch.empty(T, B, H, 128, dtype=torch.float16, device="cuda")
            st = ops.decode_values(ops.make_cache(cut, dbi, ti, book, mi, sc, spec, lead + size, bound), T, B, H, is_k, out)
            assert ops.read_status(st) == 0 and torch.equal(out.view(torch.int16), values.view(torch.int16))
    assert len(ends) == len(leads)


@pytest.mark.parametrize("is_k", [True, False])
@pytest.mark.parametrize("values", [True, False])
@pytest.mark.parametrize("T", [128, 4096])                      # a block for a pair at most; several
def test_a_staging_wait_that_runs_out(ops, is_k, values, T):
    """The waits for a block's bytes are bounded.  With the diagnostic that announces bytes which are never copied they run
    out after a few tries: the call returns, the status word says so, and the next ordinary call is correct."""
    B, H = 2, 40
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, B, H, 128, device="cuda", generator=g).half()
    hist = torch.zeros(256, dtype=torch.int64, device="cuda")
    codes, mi, sc, spec, _ = ops.quantize(x, ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN, 64, 0.05, False, min_dtype=torch.int16, hist=hist)
    book = ops.build_codebook(hist)
    bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
    bi, ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz, dtype=torch.uint8, device="cuda")
    enc = torch.empty(n, dtype=torch.uint8, device="cuda")
    total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
    size, largest = total.tolist()
    assert ops.read_status(st) == 0

    def call():
        if not values:
            return ops.decode(enc[:size], bi, ti, book, T, B, H, is_k, max_block=largest)
        out = torch.empty(T, B, H, 128, dtype=torch.float16, device="cuda")
        return out, ops.decode_values(ops.make_cache(enc, bi, ti, book, mi, sc, spec, size, largest), T, B, H, is_k, out)
    try:
        ops.decode_debug(wait_limit=8, starve=True)
        _, st = call()
        torch.cuda.synchronize()
        assert ops.read_status(st, raise_on_fatal=False) & 0x400
    finally:
        ops.decode_debug()
    out, st = call()
    want = ops.dequant(codes, mi, sc, spec) if values else codes
    assert ops.read_status(st) == 0 and torch.equal(out.view(torch.uint8), want.view(torch.uint8))
