"""How many workers the one-head attention kernel gets: its shared memory holds two decode tables and what the workers need, nothing else."""
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


def test_seven_workers_where_they_fit(ops, tmp_path):
    """Blocks of up to 6080 bytes: slots of 6112 bytes, four to a worker of 3776 bytes.  Seven workers, tables of 32 KB and 1 KB behind the slots are
    225.9 of 227 KB."""
    g = torch.Generator(device="cuda").manual_seed(1)
    T, B, H = 512, 8, 32
    caches, keep, values = [], [], []
    for is_k in (True, False):
        x = torch.randn(T, B, H, 128, device="cuda", generator=g).half()
        hist = torch.zeros(256, dtype=torch.int64, device="cuda")
        codes, mi, sc, spec, _ = ops.quantize(x, ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN, 64, 0.05, False, min_dtype=torch.int16, hist=hist)
        book = ops.build_codebook(hist)
        bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
        bi, ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz // 2, dtype=torch.int16, device="cuda")
        enc = torch.empty(n, dtype=torch.uint8, device="cuda")
        total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
        size, largest = total.tolist()
        assert ops.read_status(st) == 0 and largest <= 6080
        caches.append(ops.make_cache(enc, bi, ti, book, mi, sc, spec, size, 6080))
        keep.append((enc, bi, ti, book, mi, sc))
        values.append(ops.dequant(codes, mi, sc, spec).double())
    q = torch.randn(B, H, 128, device="cuda", generator=g).half()
    ops.attn_decode(*caches, T, B, H, q, 0.05)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        out, st = ops.attn_decode(*caches, T, B, H, q, 0.05)
        torch.cuda.synchronize()
    assert ops.read_status(st) == 0
    s = torch.einsum("bhd,tbhd->bht", q.double(), values[0]) * 0.05
    want = torch.einsum("bht,tbhd->bhd", torch.softmax(s, -1), values[1])
    assert float((out.double() - want).abs().max() / want.abs().max()) <= 1e-3
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    with open(tmp_path / "trace.json") as f:
        launches = [e["args"]["block"] for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel" and "attn_one_kernel" in e["name"]]
    if not launches:
        pytest.skip("the profiler saw no kernels")
    assert launches == [[7 * 128, 1, 1]]
