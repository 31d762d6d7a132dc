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
