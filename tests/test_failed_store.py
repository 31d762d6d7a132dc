"""Stores that fail, in part or as a whole, and stores that wait together."""
import copy
import types

import pytest
import torch

from kvcomp_b200 import _lib, ops
from kvcomp_b200.cache import kvcomp_encode
from kvcomp_b200.cache.kvcomp_cache import KVCompCache
from kvcomp_b200.cache.kvcomp_encode import KVCompCtx
from kvcomp_b200.utils.compute import QuantMode
from kvcomp_b200.utils.config import KVCompCacheConfig, KVCompCacheConfigStatic

B, H, D = 2, 3, 128


@pytest.fixture(autouse=True)
def _config():
    KVCompCacheConfigStatic.config = KVCompCacheConfig("synthetic", QuantMode("ChannelQuant"), QuantMode("TokenQuant"), 64, 64, 32, 32, 0.05, 0.1)
    yield
    KVCompCacheConfigStatic.config = None


class _Failing:
    """torch.empty whose call number `at` finds no memory."""

    def __init__(self, at):
        self.at, self.seen, self.real = at, 0, torch.empty

    def __call__(self, *a, **kw):
        self.seen += 1
        if self.seen - 1 == self.at:
            raise torch.cuda.OutOfMemoryError("no memory left")
        return self.real(*a, **kw)


def _untouched(ctx):
    return ctx.book is None and (ctx.ctx_len, ctx.compressed_ctx_len, ctx.encoded_ctx_len, len(ctx._recent), ctx._enc.n, ctx._mi.n) == (0,) * 6


def _each_failure(store):
    """store(at) with the allocations failing one after the other; returns at how many places."""
    at = 0
    while store(at):
        at += 1
    assert at >= 5
    return at


@pytest.fixture
def on_cpu(monkeypatch):
    """The calls that reach the device, on the CPU; returns what a test may set and look at."""
    d = types.SimpleNamespace(waits=[], builds=[], flags=(0, 0))
    monkeypatch.setattr(ops, "_cuda", lambda t, dtype, name: t)
    monkeypatch.setattr(ops, "wait", lambda device: d.waits.append(device))
    monkeypatch.setattr(ops.Reports, "place", staticmethod(lambda: (0, 0)))
    monkeypatch.setattr(ops.Reports, "read", staticmethod(lambda i: [1000, 500, *d.flags]))
    monkeypatch.setattr(ops, "store_at", lambda device, words, ints, rel, n_entries=0: d.builds.append(ints[4]))
    monkeypatch.setattr(ops, "rope_store", lambda x, cos, sin, out=None, first=0: x.permute(2, 0, 1, 3).contiguous())
    monkeypatch.setattr(KVCompCache, "_plain", staticmethod(lambda x: True))
    return d


@pytest.mark.parametrize("is_k", [True, False])
def test_the_next_store_builds_the_book(monkeypatch, on_cpu, is_k):
    builds = on_cpu.builds

    def store(at):
        ctx, x = KVCompCtx(is_k, B, H, D, 0.05, keep_dequantised=True), torch.zeros(200, B, H, D, dtype=torch.float16)
        failing = _Failing(at)
        with monkeypatch.context() as m:
            m.setattr(kvcomp_encode.torch, "empty", failing)
            try:
                ctx.store(x)
            except torch.cuda.OutOfMemoryError:
                pass
        failed = failing.seen > at
        if failed:
            assert _untouched(ctx), "after allocation %d" % at
            del builds[:]
            ctx.store(x)
        assert builds == [True] and ctx.ctx_len == 200 and ctx.book is not None
        del builds[:]
        return failed
    _each_failure(store)


def test_values_of_another_device_are_waited_for(on_cpu):
    """One wait is for one device: elsewhere the values' store is a call of its own."""
    x = torch.zeros(B, H, 200, D, dtype=torch.float16)
    for values in (x.to("meta"), x):
        kc, vc = KVCompCtx(True, B, H, D, 0.05, keep_dequantised=True), KVCompCtx(False, B, H, D, 0.1, keep_dequantised=True)
        del on_cpu.waits[:]
        both = KVCompCache._values_begun(kc, vc, kc.begin_heads(x, keep_codes=False), values)
        assert both == (values is x) and (kc.ctx_len, vc.ctx_len) == (200, 200 if both else 0) and on_cpu.waits == [x.device]


def test_values_wait_for_keys_that_hold_much(monkeypatch, on_cpu):
    """A first prompt's store holds nothing for its end; a later one's codes and the window that is replaced count."""
    x = torch.zeros(B, H, 200, D, dtype=torch.float16)
    kc, vc = KVCompCtx(True, B, H, D, 0.05, keep_dequantised=True), KVCompCtx(False, B, H, D, 0.1, keep_dequantised=True)
    monkeypatch.setattr(KVCompCache, "HELD", 0)
    assert KVCompCache._values_begun(kc, vc, kc.begin_heads(x, keep_codes=False), x)
    held = 192 * B * H * D + kc._recent.buf.numel() * 2
    for limit, both in ((held - 1, False), (held, True)):
        with monkeypatch.context() as m:
            m.setattr(KVCompCache, "HELD", limit)
            a, b = copy.deepcopy(kc), copy.deepcopy(vc)
            begun = a.begin_heads(x, keep_codes=False)
            assert begun.over and begun.n == 192 and begun.put_rest is None and a.held(begun) == held
            assert KVCompCache._values_begun(a, b, begun, x) == both and (a.ctx_len, b.ctx_len) == (400, 400 if both else 200)


def test_a_first_prompt_of_rows_holds_nothing(on_cpu):
    """Keys whose units are not per channel are rotated into rows first."""
    KVCompCacheConfigStatic.config.k_quant_mode = QuantMode("BlockQuant")
    x, rot = torch.zeros(B, H, 200, D, dtype=torch.float16), torch.ones(1, 200, D, dtype=torch.float16)
    kc = KVCompCtx(True, B, H, D, 0.05, keep_dequantised=True)
    begun = kc.begin_heads(x, rot, rot, keep_codes=False)
    assert begun.n == 192 and begun.n_rest == 8 and kc.held(begun) == 0 and begun.put_rest is None
    assert kc._finish(begun) is None and kc.ctx_len == 200 and kc._pending is None
    assert KVCompCtx(True, B, H, D, 0.05).store_heads(x, rot, rot).numel() == 192 * B * H * D


@pytest.mark.parametrize("flags", [(_lib.FLAG_CODE_OVERFLOW, 0), (_lib.FLAG_MIN_OVERFLOW, 0), (0, _lib.FLAG_BLOCK_LONG)])
def test_refused_keys_do_not_count(on_cpu, flags):
    """Neither they nor the values that were on their way with them; the next prompt's books are its own."""
    x = torch.zeros(B, H, 200, D, dtype=torch.float16)
    kc, vc = (KVCompCtx(is_k, B, H, D, 0.05, min_dtype=torch.int16, keep_dequantised=True) for is_k in (True, False))
    on_cpu.flags = flags
    with pytest.raises(_lib.KvcError):
        KVCompCache._values_begun(kc, vc, kc.begin_heads(x, keep_codes=False), x)
    assert _untouched(kc) and _untouched(vc) and on_cpu.builds == [True, True]
    on_cpu.flags = (0, 0)
    assert KVCompCache._values_begun(kc, vc, kc.begin_heads(x, keep_codes=False), x)
    assert on_cpu.builds == [True] * 4 and (kc.ctx_len, vc.ctx_len) == (200, 200)
    book = kc.book
    on_cpu.flags = flags                                     # a later store: what is there stays
    with pytest.raises(_lib.KvcError):
        kc.store(x.permute(2, 0, 1, 3).contiguous())
    assert kc.book is book and (kc.ctx_len, kc.compressed_ctx_len, kc.encoded_ctx_len) == (200, 192, 192) and on_cpu.builds[4:] == [False]


def test_a_stream_that_holds_nothing_is_none(on_cpu):
    """64 tokens of values wait for the other half of their Huffman block; refused keys have no unit parameters either."""
    vc, kc = KVCompCtx(False, B, H, D, 0.1), KVCompCtx(True, B, H, D, 0.05)
    vc.store(torch.zeros(64 + 32, B, H, D, dtype=torch.float16))
    assert vc.compressed_ctx_len == 64 and vc.encoded_data is None and vc.block_infos is None and vc.thread_infos is None
    assert vc.quant_min_ints.numel() == vc.quant_scales.numel() == 64
    on_cpu.flags = (_lib.FLAG_CODE_OVERFLOW, 0)
    with pytest.raises(_lib.KvcError):
        kc.store(torch.zeros(128, B, H, D, dtype=torch.float16))
    assert all(x is None for x in (kc.encoded_data, kc.block_infos, kc.thread_infos, kc.quant_min_ints, kc.quant_scales))


@pytest.mark.gpu
@pytest.mark.parametrize("heads", [True, False])
def test_a_retry_stores_what_a_first_call_would(monkeypatch, heads):
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(B, H, 300, D, device="cuda", generator=g).half()
    rows = x.permute(2, 0, 1, 3).contiguous()

    def state(ctx):
        return [ctx.ctx_len, ctx._enc.n, ctx.max_block_bytes] + \
            [t.cpu() for t in (ctx.encoded_data, ctx.block_infos, ctx.thread_infos, ctx.quant_min_ints, ctx.quant_scales, ctx.buffer, ctx.get()[0])]

    def call(ctx):
        return ctx.store_heads(x) if heads else ctx.store(rows)
    fresh = KVCompCtx(True, B, H, D, 0.05, batch_shared=False, keep_dequantised=True)
    call(fresh)
    want = state(fresh)

    def store(at):
        ctx, failing = KVCompCtx(True, B, H, D, 0.05, batch_shared=False, keep_dequantised=True), _Failing(at)
        with monkeypatch.context() as m:
            m.setattr(kvcomp_encode.torch, "empty", failing)
            try:
                call(ctx)
            except torch.cuda.OutOfMemoryError:
                pass
        if failing.seen > at:
            assert _untouched(ctx), "after allocation %d" % at
            call(ctx)
        assert all(torch.equal(a, b) if isinstance(a, torch.Tensor) else a == b for a, b in zip(state(ctx), want))
        return failing.seen > at
    _each_failure(store)


@pytest.mark.gpu
def test_a_layer_whose_keys_were_refused_takes_the_next_prompt():
    g = torch.Generator(device="cuda").manual_seed(6)
    k, v = (torch.randn(B, H, 300, D, device="cuda", generator=g).half() for _ in range(2))
    rot = {n: torch.full((1, 300, D), x, dtype=torch.float16, device="cuda") for n, x in (("cos", 1.0), ("sin", 0.0))}
    bad = k.clone()
    bad[1, 2, :, 5] = float("nan")
    cache = KVCompCache(B, H, D, 2)
    with pytest.raises(_lib.KvcError):
        cache.append(bad, v, 0, rot)
    for layer in range(2):
        cache.append(k, v, layer, rot)
    for a, b in zip((cache.k_ctx[0], cache.v_ctx[0]), (cache.k_ctx[1], cache.v_ctx[1])):
        assert a.ctx_len == b.ctx_len == 300
        for x, y in zip(*((c.encoded_data, c.block_infos, c.thread_infos, c.quant_min_ints, c.quant_scales, c.buffer, c.get()[0]) for c in (a, b))):
            assert torch.equal(x, y)


@pytest.mark.gpu
def test_a_long_prompt_behind_a_first_one_needs_little_more_memory_for_both():
    """Than its keys and its values stored one after the other."""
    heads, t = 128, 2048
    g = torch.Generator(device="cuda").manual_seed(7)

    def new(n):
        return [torch.randn(1, heads, n, D, device="cuda", generator=g).half() for _ in range(2)], \
            {name: torch.full((1, n, D), x, dtype=torch.float16, device="cuda") for name, x in (("cos", 1.0), ("sin", 0.0))}

    def together(cache, kv, rot):
        cache.append(kv[0], kv[1], 0, rot)

    def apart(cache, kv, rot):
        cache.k_ctx[0].store_heads(kv[0], rot["cos"], rot["sin"])
        cache.v_ctx[0].store_heads(kv[1])
    peaks = []
    for call in (apart, together):
        cache = KVCompCache(1, heads, D, 1)
        cache.append(*new(2000)[0], 0, new(2000)[1])         # (leaves rows in the windows)
        args = new(t)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        at = torch.cuda.memory_allocated()
        call(cache, *args)
        torch.cuda.synchronize()
        peaks.append(torch.cuda.max_memory_allocated() - at)
        del cache, args
    assert peaks[1] <= peaks[0] + (64 << 20), peaks
