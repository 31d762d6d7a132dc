"""A store is one call with one wait; keys and values of a prompt are on their way together."""
import pytest
import torch

from kvcomp_b200.utils.compute import QuantMode
from kvcomp_b200.utils.config import KVCompCacheConfig, KVCompCacheConfigStatic

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _config():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    KVCompCacheConfigStatic.config = KVCompCacheConfig("synthetic", QuantMode("ChannelQuant"), QuantMode("TokenQuant"), 64, 64, 32, 32, 0.05, 0.1)
    yield
    KVCompCacheConfigStatic.config = None


def _prompt(t, seed, H=3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k, v = (torch.randn(2, H, t, 128, device="cuda", generator=g).half() for _ in range(2))
    one, zero = (torch.full((1, t, 128), x, dtype=torch.float16, device="cuda") for x in (1.0, 0.0))
    return k, v, {"cos": one, "sin": zero}


def _state(ctx):
    return [ctx.ctx_len, ctx.compressed_ctx_len, ctx.encoded_ctx_len, ctx._enc.n, ctx.max_block_bytes] + \
        [x.cpu().clone() for x in (ctx.encoded_data, ctx.block_infos, ctx.thread_infos, ctx.quant_min_ints, ctx.quant_scales, ctx.buffer, ctx.get()[0])]


def _same(a, b):
    return all(torch.equal(x, y) if isinstance(x, torch.Tensor) else x == y for x, y in zip(a, b))


@pytest.mark.parametrize("t", [65, 200, 333, 1100])         # V's codes wait for half a Huffman block, or none do; more rows than are kept
def test_both_at_once_and_one_after_the_other(t):
    from kvcomp_b200.cache.kvcomp_cache import KVCompCache
    k, v, rot = _prompt(t, t)
    both, single = KVCompCache(2, 3, 128, 1), KVCompCache(2, 3, 128, 1)
    kc, vc = single._ctx(0, 3)
    for cut in (slice(0, t - 40), slice(t - 40, t)):         # a prompt, then more than the window holds
        r = {n: x[:, cut].contiguous() for n, x in rot.items()}
        both.append(k[:, :, cut].contiguous(), v[:, :, cut].contiguous(), 0, r)
        kc.store(k[:, :, cut].permute(2, 0, 1, 3).contiguous())
        vc.store(v[:, :, cut].permute(2, 0, 1, 3).contiguous())
        for a, b in ((both.k_ctx[0], kc), (both.v_ctx[0], vc)):
            if a.encoded_ctx_len:
                assert _same(_state(a), _state(b))


def test_keys_that_are_refused_leave_the_values_as_they_were():
    from kvcomp_b200._lib import KvcError
    from kvcomp_b200.cache.kvcomp_cache import KVCompCache
    k, v, rot = _prompt(300, 1)
    bad = k.clone()
    bad[1, 2, :, 5] = float("nan")
    cache = KVCompCache(2, 3, 128, 2)
    with pytest.raises(KvcError):
        cache.append(bad, v, 0, rot)
    vc = cache.v_ctx[0]
    assert (vc.ctx_len, vc.compressed_ctx_len, vc.encoded_ctx_len, vc._enc.n, vc.book, len(vc._recent)) == (0, 0, 0, 0, None, 0)
    cache.append(k, v, 1, rot)
    vc.store_heads(v)
    assert _same(_state(vc), _state(cache.v_ctx[1]))


@pytest.mark.parametrize("way", ["copy", "pickle"])
def test_a_copy_goes_on_by_itself(way):
    """The arenas of a first store share one allocation; a copy's and the original's do not."""
    import copy
    import pickle
    from kvcomp_b200.cache.kvcomp_cache import KVCompCache
    k, v, rot = _prompt(333, 3)
    first = {n: x[:, :200].contiguous() for n, x in rot.items()}
    rest = {n: x[:, 200:].contiguous() for n, x in rot.items()}
    want, cache = KVCompCache(2, 3, 128, 1), KVCompCache(2, 3, 128, 1)
    for c in (want, cache):
        c.append(k[:, :, :200].contiguous(), v[:, :, :200].contiguous(), 0, first)
    before = [_state(x) for x in (cache.k_ctx[0], cache.v_ctx[0])]
    ctxs = [copy.deepcopy(x) if way == "copy" else pickle.loads(pickle.dumps(x)) for x in (cache.k_ctx[0], cache.v_ctx[0])]
    want.append(k[:, :, 200:].contiguous(), v[:, :, 200:].contiguous(), 0, rest)
    for c, x in zip(ctxs, (k, v)):
        c.store(x[:, :, 200:].permute(2, 0, 1, 3).contiguous())
    assert _same(_state(ctxs[0]), _state(want.k_ctx[0])) and _same(_state(ctxs[1]), _state(want.v_ctx[0]))
    assert all(_same(a, _state(x)) for a, x in zip(before, (cache.k_ctx[0], cache.v_ctx[0])))


def test_reports_of_two_threads():
    """Each thread's stores have places of their own."""
    import threading
    from kvcomp_b200.cache.kvcomp_cache import KVCompCache
    prompts = [_prompt(200 + 64 * i, 10 + i) for i in range(4)]
    want, got = [], [None] * 4
    for k, v, rot in prompts:
        c = KVCompCache(2, 3, 128, 1)
        c.append(k, v, 0, rot)
        want.append((_state(c.k_ctx[0]), _state(c.v_ctx[0])))
    torch.cuda.synchronize()

    def body(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(10):
                k, v, rot = prompts[i]
                c = KVCompCache(2, 3, 128, 1)
                c.append(k, v, 0, rot)
            got[i] = (_state(c.k_ctx[0]), _state(c.v_ctx[0]))
    threads = [threading.Thread(target=body, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g, w in zip(got, want):
        assert g is not None and _same(g[0], w[0]) and _same(g[1], w[1])
