"""Which grouped launches decode vectors whole: those whose workers take two steps at most, one after the other, however few columns share the device.
(Whole vectors have rows of 144 bytes, the others of 32 and two tables: the launch's shared memory tells them apart.)"""
import json

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops as _ops
    return _ops


def _shared(ops, T, B, H, path, **kw):
    """Bytes of the launch's shared memory."""
    g = torch.Generator(device="cuda").manual_seed(1)
    caches, keep = [], []
    for is_k in (True, False):
        x = torch.randn(T, B, H, 128, device="cuda", generator=g).half()
        hist = torch.zeros(256, dtype=torch.int64, device="cuda")
        codes, mi, sc, spec, _ = ops.quantize(x, ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN, 64, 0.1, False, min_dtype=torch.int16, hist=hist)
        book = ops.build_codebook(hist)
        bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
        bi, ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz // 2, dtype=torch.int16, device="cuda")
        enc = torch.empty(n, dtype=torch.uint8, device="cuda")
        total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
        size, largest = total.tolist()
        assert ops.read_status(st) == 0 and largest <= 4000
        caches.append(ops.make_cache(enc, bi, ti, book, mi, sc, spec, size, 4000))
        keep.append((enc, bi, ti, book, mi, sc))
    q = torch.randn(B, H * 4, 128, device="cuda", generator=g).half()
    ops.attn_decode(*caches, T, B, H, q, 0.05, **kw)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        out, st = ops.attn_decode(*caches, T, B, H, q, 0.05, **kw)
        torch.cuda.synchronize()
    assert ops.read_status(st) == 0
    prof.export_chrome_trace(str(path / "trace.json"))
    with open(path / "trace.json") as f:
        shared = [e["args"]["shared memory"] for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel" and "attn_rows_kernel" in e["name"]]
    if not shared:
        pytest.skip("the profiler saw no kernels")
    assert len(shared) == 1
    return shared[0]


def test_many_steps_of_few_columns_are_not_brief(ops, tmp_path):
    """Eight columns without a workspace, a team of four workers for each: a step for a worker, two, and four."""
    one = dict(splits=1, workspace=False)
    step, two, four = (_shared(ops, T, 1, 8, tmp_path, **one) for T in (512, 1024, 2048))
    assert step == two > four
