"""What timed calls keep per thread (two events, a status word) does not carry over from one call to the next."""
import threading

import pytest
import torch

from kvcomp_b200.utils.compute import QuantMode
from kvcomp_b200.utils.config import KVCompCacheConfig, KVCompCacheConfigStatic

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops as _ops
    KVCompCacheConfigStatic.config = KVCompCacheConfig("synthetic", QuantMode("ChannelQuant"), QuantMode("TokenQuant"),
                                                       64, 128, 0, 0, 0.05, 0.1)
    yield _ops
    KVCompCacheConfigStatic.config = None


def _in_a_new_thread(fn):
    """A thread keeps its own: fn's first timed call is the thread's first."""
    raised = []

    def body():
        try:
            fn()
        except BaseException as e:
            raised.append(e)
    t = threading.Thread(target=body)
    t.start()
    t.join()
    if raised:
        raise raised[0]


def _context(seed=0):
    from kvcomp_b200.cache.kvcomp_encode import KVCompCtx
    c = KVCompCtx(False, 1, 2, 128, 0.1, batch_shared=False, min_dtype=torch.int16)
    c.store(torch.randn(256, 1, 2, 128, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).half())
    return c


def _every_timed_call(ops, c):
    from kvcomp_b200 import kvcomp_cuda
    c.get()
    codes, _ = c.get_decode_quant_ints()
    c.mat_vec_mul(torch.rand(1, 2, 256, device="cuda").half())
    out = torch.empty_like(codes)
    kvcomp_cuda.v_entropy_decode_cuda_export(c.encoded_data, c.block_infos, c.thread_infos, c.decode_codebook, out, 2, 128)
    assert torch.equal(out, codes)


@pytest.mark.parametrize("inference_first", [True, False])
def test_inference_mode_and_ordinary_calls_in_one_thread(ops, inference_first):
    def body():
        c = _context()
        for inference in (inference_first, not inference_first, inference_first):
            with torch.inference_mode(inference):
                _every_timed_call(ops, c)
    _in_a_new_thread(body)


@pytest.mark.parametrize("side_stream", [False, True])
def test_flags_of_a_call_that_ended_early_are_not_the_next_ones(ops, side_stream):
    def body():
        c = _context()
        for raised in (KeyError, ops.KvcError):                # between the launches and end(); by end() itself
            with torch.cuda.stream(torch.cuda.Stream() if side_stream else torch.cuda.current_stream()):
                with pytest.raises(raised):
                    with ops.TimedCall.on(c.device) as call:
                        torch.cuda._sleep(100_000_000)         # the call's kernels are still at work when it ends
                        call.status.fill_(ops._lib.FLAG_BAD_STREAM)
                        if raised is KeyError:
                            raise KeyError
                        call.end("decode")
            _every_timed_call(ops, c)
            assert int(ops.TimedCall.on(c.device).status.item()) == 0
    _in_a_new_thread(body)


def test_a_call_that_raises_behind_its_launch(ops, monkeypatch):
    def body():
        c, other = _context(), _context(1)
        bad = c._ti.buf.clone()
        c._ti.buf.fill_(-1)                                # every vector but a block's first begins outside its block
        c._pending = torch.zeros(1, 1, 2, 128, dtype=torch.uint8, device="cuda")

        def fail(*a, **kw):
            raise MemoryError("no room")
        monkeypatch.setattr(ops, "dequant", fail)
        with pytest.raises(MemoryError):
            c.get()
        monkeypatch.undo()
        _every_timed_call(ops, other)
        c._ti.buf, c._pending = bad, None
        _every_timed_call(ops, c)
    _in_a_new_thread(body)


def test_the_first_call_of_a_thread_waits_for_its_own_stream_only(ops):
    def body():
        ops.new_status("cuda:0")                               # memory for both words is at hand
        torch.empty(1, dtype=torch.int32, pin_memory=True)
        torch.cuda.synchronize()
        other, done = torch.cuda.Stream(), torch.cuda.Event()
        with torch.cuda.stream(other):
            torch.cuda._sleep(1_000_000_000)                   # half a second
            done.record()
        ops.TimedCall.on(torch.device("cuda", 0))
        assert not done.query()
        done.synchronize()
    _in_a_new_thread(body)
