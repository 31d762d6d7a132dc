"""Grouped attention by the ways a book can be decoded: two codes in every window, in all but a few (lanes fall behind, catch up, or take
their 32 symbols again), one symbol per lookup, and either with codes beyond the window; launches of a step per worker decode whole vectors."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops as _ops
    return _ops


# symbol frequencies; what the book has to be: (codes beyond the window, windows with fewer than two codes: lowest, highest)
BOOKS = {
    "pairs": ([1.0] * 8, (0, 0, 0)),
    "misses": ([2.0 ** -abs(i - 7) for i in range(15)], (0, 1, 60)),
    "singles": ([1.0] * 128, (0, 4096, 4096)),
    "pairs_long": ([2.0 ** -(i + 1) for i in range(18)], (1, 1, 100)),
    "singles_long": ([1.0] * 100 + [2.0 ** -i for i in range(1, 12)], (1, 101, 4096)),
}


def _codes(kind, shape, is_k, g):
    p = torch.tensor(BOOKS[kind][0], device="cuda")
    n = shape[0] * shape[1] * shape[2] * shape[3]
    edges = (p.double() / p.double().sum()).cumsum(0)
    codes = torch.searchsorted(edges, torch.rand(n, dtype=torch.float64, device="cuda", generator=g)).clamp_(max=len(p) - 1).to(torch.uint8).view(shape)
    rare = len(p) - 1
    # vectors of nothing but the rarest symbol, and some with a run of it at every place of a round: lanes lag by 1, 2, .. symbols.  (They are few
    # enough for the book to keep its long codes.)
    for i in range(1, 13):
        if is_k:
            codes[i * 7 % shape[0], 0, 0, 9 * i:9 * i + i] = rare
        else:
            codes[9 * i:9 * i + i, 0, 0, 5 * i] = rare
    if is_k:
        codes[5, -1, -1] = rare
    else:
        codes[128:256, -1, -1, 77] = rare
    return codes


def _cache(ops, kind, shape, is_k, g):
    T, B, H, _ = shape
    codes = _codes(kind, shape, is_k, g)
    book = ops.build_codebook(torch.bincount(codes.flatten().int(), minlength=256))
    escape, low, high = BOOKS[kind][1]
    lone = book.host()[32:36].view(torch.int32).item()
    assert book.header()["escape"] == escape and lone >> 16 == 0x4b56 and low <= (lone & 0xffff) <= high, (book.header(), hex(lone))
    spec = ops.qspec(ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN, False, B, H, 128, 64)
    units = spec.units(T, B, H, 128)
    mi = torch.randint(-300, 300, (units,), device="cuda", generator=g).to(torch.int16)
    sc = (0.002 + 0.03 * torch.rand(units, device="cuda", generator=g)).half()
    if not is_k:
        sc[::5] = -sc[::5]                                 # what a caller of the C interface may hand over
    bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
    bi, ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz // 2, dtype=torch.int16, device="cuda")
    enc = torch.empty(2 * n, dtype=torch.uint8, device="cuda")
    total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
    size, largest = total.tolist()
    assert ops.read_status(st) & ~ops._lib.FLAG_VECTOR_LONG == 0         # (vectors of long codes only: longer than the reference's scratch, stored all the same)
    u = (torch.arange(T, device="cuda") // spec.tok_div)[:, None, None, None] * spec.sj + torch.arange(B, device="cuda")[None, :, None, None] * spec.sb + \
        torch.arange(H, device="cuda")[None, None, :, None] * spec.sh + torch.arange(128, device="cuda")[None, None, None, :] * spec.sc
    exact = (codes.double() + mi[u].double()) * sc[u].double()
    return ops.make_cache(enc, bi, ti, book, mi, sc, spec, size, largest), exact, (enc, bi, ti, book, mi, sc)


@pytest.mark.parametrize("G", [2, 4, 8])
@pytest.mark.parametrize("kk,vk", [("pairs", "misses"), ("misses", "pairs"), ("singles", "misses"), ("pairs_long", "singles"), ("singles_long", "pairs_long"),
                                   ("misses", "singles_long")])
@pytest.mark.parametrize("T,B,H,rounds", [(1536, 16, 4, None), (6144, 16, 4, 4), (256, 2, 1, 0)])    # (rounds of steps that the device's workers take)
def test_ways(ops, G, kk, vk, T, B, H, rounds):
    workers = 5 * torch.cuda.get_device_properties(0).multi_processor_count
    steps = B * H * T // 128
    if rounds == 0:
        assert steps <= workers                            # vectors are decoded whole
    elif rounds:
        assert steps > rounds * workers                    # by pairs and singles; items of several steps
    g = torch.Generator(device="cuda").manual_seed(T + G)
    kc, ke, keep_k = _cache(ops, kk, (T, B, H, 128), True, g)
    vc, ve, keep_v = _cache(ops, vk, (T, B, H, 128), False, g)
    q = torch.randn(B, H * G, 128, device="cuda", generator=g).half()
    scaling = 0.25 / math.sqrt(128)
    out, st = ops.attn_decode(kc, vc, T, B, H, q, scaling)
    assert ops.read_status(st) == 0
    s = torch.einsum("bhgd,tbhd->bhgt", q.double().view(B, H, G, 128), ke) * scaling
    want = torch.einsum("bhgt,tbhd->bhgd", torch.softmax(s, -1), ve).reshape(B, H * G, 128)
    # 1e-3 of the largest output, as for the attention everywhere (weights of 16 bits, fp16 outputs)
    assert float((out.double() - want).abs().max() / want.abs().max()) <= 1e-3
