"""Prompts quantised where their projections left them (kvc_quantize_heads) against the rotated and transposed rows through
kvc_quantize: the same bits; and the stores that quantise them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops as _ops
    return _ops


def _prompt(B, H, t, seed, spread=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = (torch.randn(B, H, t, 128, device="cuda", generator=g) * spread +
         torch.randn(B, H, 1, 128, device="cuda", generator=g) * 3).half()
    ang = torch.rand(B, t, 128, device="cuda", generator=g) * 6.28
    return x, ang.cos().half(), ang.sin().half()


@pytest.mark.parametrize("mode,block,B,H,T,more,rope", [
    ("ChannelQuant", 64, 1, 1, 64, 0, "each"), ("ChannelQuant", 64, 2, 5, 192, 13, "each"), ("ChannelQuant", 64, 3, 8, 1024, 1, "one"),
    ("ChannelQuant", 128, 2, 3, 256, 77, "one"), ("ChannelQuant", 128, 1, 32, 1280, 0, None), ("ChannelQuant", 64, 16, 8, 640, 5, None),
    ("TokenQuant", 64, 1, 1, 3, 0, None), ("TokenQuant", 64, 2, 5, 64, 7, None), ("TokenQuant", 64, 2, 8, 129, 0, None),
    ("TokenQuant", 64, 3, 13, 130, 3, None), ("TokenQuant", 64, 1, 32, 700, 1, None), ("TokenQuant", 64, 2, 40, 66, 0, None),
    ("TokenQuant", 64, 1, 64, 65, 0, None), ("VectorQuant", 64, 2, 3, 67, 2, None), ("VectorQuant", 64, 1, 33, 64, 0, None),
])
def test_prompt_in_place_equals_rows(ops, mode, block, B, H, T, more, rope):
    m = ops.MODES[mode]
    assert ops.quantize_heads_fits(m, False, T, B, H, 128, block)
    for seed, spread, rel in ((1, 1.0, 0.05), (2, 300.0, 0.2), (3, 1e-6, 0.003)):      # the last two leave the packed arithmetic
        x, cos, sin = _prompt(B, H, T + more, seed, spread)
        x[0, 0, :T, 5] = 1.5                                                           # a constant channel
        cos, sin = (None, None) if rope is None else (cos, sin) if rope == "each" else (cos[:1].contiguous(), sin[:1].contiguous())
        rows = ops.rope_store(x, cos, sin)
        spec = ops.qspec(m, False, B, H, 128, block)
        n = spec.units(T, B, H, 128)
        for dt in (torch.int8, torch.int16):
            hist, hist2 = (torch.zeros(256, dtype=torch.int64, device="cuda") for _ in range(2))
            want, mi, sc, _, st = ops.quantize(rows[:T].contiguous(), m, block, rel, False, min_dtype=dt, hist=hist)
            mi2, sc2, st2 = torch.empty_like(mi), torch.empty_like(sc), ops.new_status(x.device)
            got = ops.quantize_heads(x, T, cos, sin, m, block, rel, False, mi2, sc2, hist2, st2)
            assert torch.equal(sc.view(torch.int16), sc2.view(torch.int16)) and torch.equal(mi, mi2) and mi2.numel() == n
            assert torch.equal(want, got) and torch.equal(hist, hist2)
            assert int(st.item()) == int(st2.item())
        if more:
            assert torch.equal(ops.rope_store(x, cos, sin, first=T), rows[T:])


@pytest.mark.parametrize("mode,block,rope", [("ChannelQuant", 64, "each"), ("ChannelQuant", 64, None), ("ChannelQuant", 128, None),
                                             ("TokenQuant", 64, None), ("VectorQuant", 64, None)])
@pytest.mark.parametrize("special", [float("nan"), float("inf"), float("-inf"), -0.0, 65504.0])
def test_prompt_of_special_values_equals_rows(ops, mode, block, rope, special):
    m, (B, H, T) = ops.MODES[mode], (2, 5, 256)
    for where in ("channel", "token", "head", "half a block", "one"):
        x, cos, sin = _prompt(B, H, T, 1)
        at = {"channel": (1, 2, slice(None), 77), "token": (1, slice(None), 130), "head": (0, 4), "one": (0, 1, 3, 100),
              "half a block": (1, 0, slice(0, block // 2), slice(None))}[where]
        x[at] = special
        cos, sin = (None, None) if rope is None else (cos, sin)
        rows = ops.rope_store(x, cos, sin)
        hist, hist2 = (torch.zeros(256, dtype=torch.int64, device="cuda") for _ in range(2))
        want, mi, sc, _, st = ops.quantize(rows, m, block, 0.05, False, min_dtype=torch.int16, hist=hist)
        mi2, sc2, st2 = torch.empty_like(mi), torch.empty_like(sc), ops.new_status(x.device)
        got = ops.quantize_heads(x, T, cos, sin, m, block, 0.05, False, mi2, sc2, hist2, st2)
        assert int(st.item()) == int(st2.item()), where
        assert torch.equal(sc.view(torch.int16), sc2.view(torch.int16)) and torch.equal(mi, mi2), where
        assert torch.equal(want, got) and torch.equal(hist, hist2), where


def test_units_that_need_rows_are_refused(ops):
    fits = ops.quantize_heads_fits
    assert not fits(ops.MODE_TOKEN, True, 64, 2, 8, 128, 64) and fits(ops.MODE_TOKEN, True, 64, 1, 8, 128, 64)
    assert not fits(ops.MODE_TOKEN, False, 64, 2, 65, 128, 64) and not fits(ops.MODE_CHANNEL, False, 192, 2, 8, 128, 192)
    assert not fits(ops.MODE_BLOCK, False, 64, 2, 8, 128, 64) and not fits(ops.MODE_CHANNEL, False, 64, 2, 8, 64, 64)


@pytest.mark.parametrize("is_k", [True, False])
@pytest.mark.parametrize("heads_first", [True, False])
def test_a_prompt_is_read_when_the_store_returns(ops, monkeypatch, is_k, heads_first):
    from kvcomp_b200.cache.kvcomp_encode import KVCompCtx
    from kvcomp_b200.utils.compute import QuantMode
    from kvcomp_b200.utils.config import KVCompCacheConfig, KVCompCacheConfigStatic
    monkeypatch.setattr(KVCompCacheConfigStatic, "config", KVCompCacheConfig(
        "synthetic", QuantMode("ChannelQuant"), QuantMode("TokenQuant"), 64, 64, 32, 32, 0.05, 0.1))
    ctx = KVCompCtx(is_k, 2, 4, 128, 0.1, batch_shared=False, min_dtype=torch.int16, keep_dequantised=True)
    x, cos, sin = _prompt(2, 4, 300, 1)
    cos, sin = (cos, sin) if is_k and heads_first else (None, None)
    rows = ops.rope_store(x, cos, sin)
    want = rows.clone()
    dequant = ops.dequant

    def late(*a, **kw):                                        # what the store launches behind its wait comes late
        torch.cuda._sleep(200_000_000)
        return dequant(*a, **kw)
    monkeypatch.setattr(ops, "dequant", late)
    torch.empty_like(x).zero_()                                # (a kernel's first launch may wait for the device)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        if heads_first:
            ctx.store_heads(x, cos, sin)
        else:
            ctx.store(rows)
    for t in (x, rows) + ((cos, sin) if cos is not None else ()):
        t.zero_()                                              # on the tensors' own stream: they are the caller's again
    torch.cuda.synchronize()
    live = len(ctx.buffer)
    assert 32 <= live < 300 and torch.equal(ctx.buffer, want[-live:])


@pytest.mark.parametrize("mode,block,H", [("ChannelQuant", 64, 3), ("ChannelQuant", 128, 8), ("TokenQuant", 64, 8), ("VectorQuant", 64, 33)])
@pytest.mark.parametrize("rel", [0.2, 0.033, 0.03, 0.004])      # codes below 32 alone, around it, up to 250
def test_prompt_counts_start_from_zero(ops, mode, block, H, rel):
    """Launch behind launch, each over the counters that the one before left in shared memory."""
    m = ops.MODES[mode]
    x, _, _ = _prompt(2, H, 512, 7)
    n = ops.qspec(m, False, 2, H, 128, block).units(512, 2, H, 128)
    mi, sc = torch.empty(n, dtype=torch.int16, device="cuda"), torch.empty(n, dtype=torch.float16, device="cuda")
    for _ in range(3):
        hist = torch.zeros(256, dtype=torch.int64, device="cuda")
        codes = ops.quantize_heads(x, 512, None, None, m, block, rel, False, mi, sc, hist, ops.new_status(x.device))
        assert torch.equal(hist, torch.bincount(codes.view(-1), minlength=256))
