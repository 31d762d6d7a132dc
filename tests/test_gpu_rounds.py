"""Attention over more columns than the device has workers, and over equal runs that go in a few rounds: how many workers an SM
gets and whether they share columns follows from the number of rounds (148 SMs: 1036 workers with one head, 740 with four, 592 with eight)."""
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


def _cache(ops, x, is_k, rel):
    T, B, H, _ = x.shape
    hist = torch.zeros(256, dtype=torch.int64, device="cuda")
    codes, mi, sc, spec, _ = ops.quantize(x, ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN, 64, rel, False, min_dtype=torch.int16, hist=hist)
    book = ops.build_codebook(hist)
    bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
    bi, ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz // 2, dtype=torch.int16, device="cuda")
    enc = torch.empty(n, dtype=torch.uint8, device="cuda")
    total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
    size, largest = total.tolist()
    assert ops.read_status(st) == 0
    return ops.make_cache(enc, bi, ti, book, mi, sc, spec, size, largest), ops.dequant(codes, mi, sc, spec), (enc, bi, ti, book, mi, sc)


@pytest.mark.parametrize("B,Hkv,G,T,Tr", [
    (37, 28, 1, 256, 0), (61, 17, 1, 128, 0), (61, 17, 1, 512, 9), (40, 32, 1, 640, 0), (33, 64, 1, 256, 0), (6, 32, 1, 1024, 0), (9, 4, 1, 2048, 0),
    (37, 20, 4, 256, 0), (57, 13, 4, 384, 0), (57, 13, 4, 256, 130), (25, 32, 4, 512, 0), (593, 1, 8, 256, 0), (100, 8, 3, 128, 0)])
def test_columns_and_runs_in_rounds(ops, B, Hkv, G, T, Tr):
    g = torch.Generator(device="cuda").manual_seed(B * T + G)
    k, v = (torch.randn(T + Tr, B, Hkv, 128, device="cuda", generator=g).half() for _ in range(2))
    q = torch.randn(B, Hkv * G, 128, device="cuda", generator=g).half()
    kc, ke, keep_k = _cache(ops, k[:T].contiguous(), True, 0.05)
    vc, ve, keep_v = _cache(ops, v[:T].contiguous(), False, 0.1)
    kt, vt = (k[T:].contiguous(), v[T:].contiguous()) if Tr else (None, None)
    ke, ve = torch.cat([ke, k[T:]]), torch.cat([ve, v[T:]])
    want = torch.empty(B, Hkv * G, 128, dtype=torch.float64, device="cuda")
    for b in range(B):
        s = torch.einsum("hgd,thd->hgt", q[b].double().view(Hkv, G, 128), ke[:, b].double()) / math.sqrt(128)
        want[b] = torch.einsum("hgt,thd->hgd", torch.softmax(s, -1), ve[:, b].double()).reshape(Hkv * G, 128)
    # 1e-3 of the largest output, as for the attention everywhere: weights of 16 bits, fp16 outputs, and here values rounded to fp16
    for splits in (0, 1, 2, 3, 5):
        for kw in ({}, {"workspace": False}) if splits == 1 else ({},):
            out, st = ops.attn_decode(kc, vc, T, B, Hkv, q, 1.0 / math.sqrt(128), kt, vt, splits=splits, **kw)
            assert ops.read_status(st) == 0
            assert float((out.double() - want).abs().max() / want.abs().max()) <= 1e-3, (splits, kw)
