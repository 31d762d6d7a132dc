"""Grouped attention at scores far beyond those of trained models: fp16 queries and keys are finite up to scores of 1e11, where a rounding of the score
is more than a weight's whole range.  A clear winner's weight stays 1 whatever the score and the sign of its V scale, and rows behind the
compressed part weigh what equal scores in it weigh."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

SCALING = 0.25                            # (a power of two: scores of one channel are exact in 32 bits)


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops as _ops
    return _ops


def _spec(ops, shape, is_k):
    T, B, H, _ = shape
    spec = ops.qspec(ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN, False, B, H, 128, 64)
    return spec, spec.units(T, B, H, 128)


def _cache(ops, codes, is_k, mi, sc):
    """A cache of given codes and units (K per channel, V per token); its values in 64 bits."""
    T, B, H, _ = codes.shape
    spec, units = _spec(ops, codes.shape, is_k)
    assert mi.numel() == sc.numel() == units
    u = (torch.arange(T, device="cuda") // spec.tok_div)[:, None, None, None] * spec.sj + torch.arange(B, device="cuda")[None, :, None, None] * spec.sb + \
        torch.arange(H, device="cuda")[None, None, :, None] * spec.sh + torch.arange(128, device="cuda")[None, None, None, :] * spec.sc
    book = ops.build_codebook(torch.bincount(codes.flatten().int(), minlength=256))
    bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
    bi, ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz // 2, dtype=torch.int16, device="cuda")
    enc = torch.empty(2 * n, dtype=torch.uint8, device="cuda")
    total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
    size, largest = total.tolist()
    assert ops.read_status(st) == 0
    return ops.make_cache(enc, bi, ti, book, mi, sc, spec, size, largest), (codes.double() + mi[u].double()) * sc[u].double(), (enc, bi, ti, book, mi, sc)


def _keys(ops, codes, mi, sc):
    """The same unit for every 64 tokens; mi and sc: [128]."""
    n = _spec(ops, codes.shape, True)[1] // 128
    return _cache(ops, codes, True, mi.repeat(n), sc.repeat(n))


def _values(ops, shape, g, least, sign=1):
    codes = torch.randint(0, 15, shape, device="cuda", generator=g).to(torch.uint8)
    n = _spec(ops, shape, False)[1]
    return _cache(ops, codes, False, torch.randint(least, 30, (n,), device="cuda", generator=g).to(torch.int16),
                  sign * (0.002 + 0.03 * torch.rand(n, device="cuda", generator=g)).half())


def _shape(long):
    """A launch with a step per worker at most, and one whose workers take several (five workers on an SM, steps of 128 tokens)."""
    B, H = 16, 4
    steps = 2
    if long:
        workers = 5 * torch.cuda.get_device_properties(0).multi_processor_count
        steps = 4 * workers // (B * H) + 1
    return 128 * steps, B, H


@pytest.mark.parametrize("long", [False, True])
@pytest.mark.parametrize("G", [2, 4, 8])
@pytest.mark.parametrize("score,negative", [(2e4, False), (2e5, False), (-2e5, False), (1e6, False), (-1e6, False), (1e9, False), (-1e9, False),
                                            (1e3, True), (1e4, True), (-1e5, True), (1e9, True)])
def test_one_token_wins(ops, G, long, score, negative):
    g = torch.Generator(device="cuda").manual_seed(G)
    T, B, H = _shape(long)
    a = 16.0 if abs(score) < 1e8 else 4096.0
    sc = torch.full((128,), abs(score) / (448 * SCALING * a), device="cuda").half()
    sign = torch.randint(0, 2, (B, H, G, 128), device="cuda", generator=g)
    codes = torch.randint(0, 8, (T, B, H, 128), device="cuda", generator=g).to(torch.uint8)
    win = torch.stack([torch.randperm(T, device="cuda", generator=g)[:G] for _ in range(B * H)]).view(B, H, G)
    for i in range(G):                                     # seven where the head's query is positive, zero where it is negative
        codes.scatter_(0, win[None, :, :, i, None].expand(1, B, H, 128), (7 * sign[:, :, i]).to(torch.uint8)[None])
    mi = torch.zeros(128, device="cuda", dtype=torch.int16)
    if score < 0:                                          # one channel takes every token's score below zero
        mi[127] = -1000
        sign[..., 127] = 1
    q = (a * (2 * sign - 1)).half().reshape(B, H * G, 128)
    kc, ke, keep_k = _keys(ops, codes, mi, sc)
    vc, ve, keep_v = _values(ops, codes.shape, g, -30, -1 if negative else 1)
    s = torch.einsum("bhgd,tbhd->bhgt", q.double().view(B, H, G, 128), ke) * SCALING
    top = s.topk(2, dim=-1)
    assert torch.equal(top.indices[..., 0], win) and float((top.values[..., 0] - top.values[..., 1]).min()) > 100 + 1e-3 * abs(score)
    assert 0.5 * abs(score) < abs(float(top.values.abs().mean()))
    want = ve.permute(1, 2, 0, 3).gather(2, win[..., None].expand(B, H, G, 128)).reshape(B, H * G, 128)
    for kw in (dict(), dict(splits=1, workspace=False)):
        out, st = ops.attn_decode(kc, vc, T, B, H, q, SCALING, **kw)
        assert ops.read_status(st) == 0
        # the winner's value in 16-bit fixed point (half a step times codes below 16) and fp16
        assert float((out.double() - want).abs().max() / want.abs().max()) <= 1e-3, kw


@pytest.mark.parametrize("long", [False, True])
@pytest.mark.parametrize("G", [2, 4, 8])
@pytest.mark.parametrize("where,value", [("q", math.inf), ("q", math.nan), ("k", math.inf), ("k", math.nan), ("v", math.inf), ("v", math.nan)])
def test_what_is_not_finite_reaches_the_output(ops, G, long, where, value):
    """Of its sequence and of no other."""
    g = torch.Generator(device="cuda").manual_seed(G)
    T, B, H = _shape(long)
    codes = torch.randint(0, 8, (T, B, H, 128), device="cuda", generator=g).to(torch.uint8)
    kc, ke, keep_k = _keys(ops, codes, torch.full((128,), -3, device="cuda", dtype=torch.int16), torch.full((128,), 0.1, device="cuda").half())
    vc, ve, keep_v = _values(ops, codes.shape, g, -30)
    q = torch.randn(B, H * G, 128, device="cuda", generator=g).half()
    clean, st = ops.attn_decode(kc, vc, T, B, H, q, SCALING)
    assert ops.read_status(st) == 0 and torch.isfinite(clean).all()
    if where == "q":
        q[3, :, 7] = value
    else:                                                  # sequence 3's last units: keys of the last block, values of the last token
        spec = _spec(ops, codes.shape, where == "k")[0]
        t = (T - 1) // spec.tok_div
        at = t * spec.sj + 3 * spec.sb + torch.arange(H, device="cuda") * spec.sh + (7 * spec.sc if where == "k" else 0)
        (keep_k if where == "k" else keep_v)[5][at] = value
    out, st = ops.attn_decode(kc, vc, T, B, H, q, SCALING)
    assert ops.read_status(st) == 0
    assert not torch.isfinite(out[3]).any()
    rest = [b for b in range(B) if b != 3]
    assert torch.equal(out[rest], clean[rest])


@pytest.mark.parametrize("long", [False, True])
@pytest.mark.parametrize("G", [2, 4, 8])
@pytest.mark.parametrize("q0", [10.0, 1000.0, 4097.0, 60000.0])
@pytest.mark.parametrize("kw", [dict(), dict(splits=4), dict(splits=1, workspace=False)])
def test_equal_scores_weigh_the_same(ops, G, long, q0, kw):
    """One channel of the query is not zero, and there all keys are equal: every token has the same score, which 32 bits hold."""
    g = torch.Generator(device="cuda").manual_seed(G)
    T, B, H = _shape(long)
    Tr = 200
    codes = torch.randint(0, 8, (T, B, H, 128), device="cuda", generator=g).to(torch.uint8)
    codes[..., 5] = 100
    kc, ke, keep_k = _keys(ops, codes, torch.zeros(128, device="cuda", dtype=torch.int16), torch.ones(128, device="cuda").half())
    vc, ve, keep_v = _values(ops, codes.shape, g, 1)
    kt = torch.randn(Tr, B, H, 128, device="cuda", generator=g).half()
    kt[..., 5] = 100.0
    vt = (-5.0 * T / Tr * (0.5 + torch.rand(Tr, B, H, 128, device="cuda", generator=g))).half()      # (as heavy as the compressed part, the other way)
    q = torch.zeros(B, H * G, 128, device="cuda").half()
    q[..., 5] = q0
    want = ((ve.sum(0) + vt.double().sum(0)) / (T + Tr)).repeat_interleave(G, 1)
    out, st = ops.attn_decode(kc, vc, T, B, H, q, SCALING, kt, vt, **kw)
    assert ops.read_status(st) == 0
    # 1e-3 of the largest output, as for the attention everywhere (weights of 16 bits, fp16 outputs)
    assert float((out.double() - want).abs().max() / want.abs().max()) <= 1e-3
