"""A decode step whose tokens are not rows of the cache's recent window is refused before anything is written."""
import pytest
import torch

from kvcomp_b200._lib import KvcError
from kvcomp_b200.utils.compute import QuantMode
from kvcomp_b200.utils.config import KVCompCacheConfig, KVCompCacheConfigStatic

pytestmark = pytest.mark.gpu


@pytest.fixture()
def cache():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200.cache.kvcomp_cache import KVCompCache
    KVCompCacheConfigStatic.config = KVCompCacheConfig("synthetic", QuantMode("ChannelQuant"), QuantMode("TokenQuant"),
                                                       64, 64, 32, 32, 0.05, 0.1)
    yield KVCompCache(2, 4, 128, 1)
    KVCompCacheConfigStatic.config = None


def _append(cache, B, H, t, D, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k, v = (torch.randn(B, H, t, D, device="cuda", generator=g).half() for _ in range(2))
    cs = torch.ones(1, t, D, device="cuda", dtype=torch.float16)
    cache.append(k, v, 0, {"cos": cs, "sin": torch.zeros_like(cs)})
    return k, v


@pytest.mark.parametrize("first", [0, 5, 150])                # a fresh cache, a window alone, streams and a window
@pytest.mark.parametrize("B,H,D", [(3, 4, 128), (1, 4, 128), (2, 5, 128), (2, 2, 128), (2, 4, 256), (2, 4, 64), (4, 2, 128), (1, 8, 128)])
def test_other_shapes_are_refused(cache, first, B, H, D):
    if first:
        _append(cache, 2, 4, first, 128)
    else:
        cache._ctx(0, 4)
    kc, vc = cache.k_ctx[0], cache.v_ctx[0]
    before = [(c.ctx_len, len(c._recent), c.compressed_ctx_len, None if c.buffer is None else c.buffer.clone()) for c in (kc, vc)]
    for t in (1, 3):
        with pytest.raises(KvcError):
            _append(cache, B, H, t, D, seed=1)
    for c, (n, live, comp, rows) in zip((kc, vc), before):
        assert (c.ctx_len, len(c._recent), c.compressed_ctx_len) == (n, live, comp)
        assert rows is None or torch.equal(c.buffer, rows)
    k, v = _append(cache, 2, 4, 1, 128, seed=2)               # and goes on
    assert torch.equal(kc.buffer[-1], k[:, :, 0]) and torch.equal(vc.buffer[-1], v[:, :, 0])


def test_a_window_set_to_other_rows_is_refused(cache):
    _append(cache, 2, 4, 5, 128)
    kc = cache.k_ctx[0]
    rows = kc.buffer
    spare = torch.zeros(64, 1, 4, 128, device="cuda", dtype=torch.float16)
    kc.buffer = spare
    kc._recent.hi = 5                                         # with room behind its rows
    with pytest.raises(KvcError):
        _append(cache, 2, 4, 1, 128)
    assert not spare.any() and kc.ctx_len == 5
    kc.buffer = rows.clone()
    k, _ = _append(cache, 2, 4, 1, 128, seed=3)
    assert torch.equal(kc.buffer[:5], rows) and torch.equal(kc.buffer[5], k[:, :, 0])
