"""The library in a process with more than one CUDA context on a device (a host that owns its contexts through the
driver interface): what it remembers of its kernels belongs to a context, not to the device."""
import ctypes as C
import multiprocessing as mp

import pytest
import torch

pytestmark = pytest.mark.gpu


class _Context:
    """A second context of device 0, current while the block runs; copies tensors in and out of it."""

    def __enter__(self):
        self.cu = C.CDLL("libcuda.so.1")
        dev, self.ctx = C.c_int(), C.c_void_p()
        self._ok(self.cu.cuInit(0))
        self._ok(self.cu.cuDeviceGet(C.byref(dev), 0))
        self._ok(self.cu.cuCtxCreate_v2(C.byref(self.ctx), 0, dev))
        return self

    def _ok(self, rc):
        assert rc == 0, "driver call failed with %d" % rc

    def put(self, host):
        host = host.contiguous()
        p = C.c_uint64()
        n = max(host.numel() * host.element_size(), 16)
        self._ok(self.cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(n)))
        self._ok(self.cu.cuMemcpyHtoD_v2(p, C.c_void_p(host.data_ptr()), C.c_size_t(host.numel() * host.element_size())))
        return p.value

    def get(self, p, like):
        out = torch.empty_like(like, device="cpu")
        self._ok(self.cu.cuCtxSynchronize())
        self._ok(self.cu.cuMemcpyDtoH_v2(C.c_void_p(out.data_ptr()), C.c_uint64(p), C.c_size_t(out.numel() * out.element_size())))
        return out

    def __exit__(self, *exc):
        self._ok(self.cu.cuCtxDestroy_v2(self.ctx))          # the primary context is current again
        return False


def _second_context(entry, q):
    try:
        from kvcomp_b200 import _lib, ops
        from kvcomp_b200.synth import make_kv
        lib = _lib.load()
        T, B, Hkv, Hq = 512, 1, 2, 4
        k, v, query = make_kv(T, B, Hkv, 128, seed=5, device="cuda", Hq=Hq)
        caches, host = [], []
        for x, is_k, mode in ((k, True, ops.MODE_CHANNEL), (v, False, ops.MODE_TOKEN)):
            hist = torch.zeros(256, dtype=torch.int64, device="cuda")
            codes, mi, sc, spec, _ = ops.quantize(x, mode, 64, 0.05, False, min_dtype=torch.int16, hist=hist)
            book = ops.build_codebook(hist)
            bsz, tsz, _, cap = ops.buffer_sizes(T, B * Hkv * 128, is_k)
            bi, ti = torch.zeros(bsz, dtype=torch.uint8, device="cuda"), torch.zeros(tsz // 2, dtype=torch.int16, device="cuda")
            enc = torch.zeros(cap, dtype=torch.uint8, device="cuda")
            total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
            n, biggest = (int(w) for w in total.tolist())
            ops.read_status(st)
            caches.append((ops.make_cache(enc, bi, ti, book, mi, sc, spec, n, biggest), (enc, bi, ti, book, mi, sc)))
            host.append(([t.cpu() for t in (enc, bi, ti, book.blob, mi, sc)], spec, n, biggest))
        (kc, _), (vc, keep_v) = caches
        out, codes = torch.empty(B, Hq, 128, dtype=torch.float16, device="cuda"), torch.empty(T, B, Hkv, 128, dtype=torch.uint8, device="cuda")

        def call(kc, vc, query, out, codes, status, ws, ws_bytes):
            if entry == "decode":
                _lib.check(lib.kvc_decode_bounded(vc.encoded, vc.encoded_bytes, vc.block_info, vc.thread_info, vc.book, T, B * Hkv, 0,
                                                  vc.max_block_bytes, codes, status, None), "kvc_decode_bounded")
            elif entry == "attn":
                _lib.check(lib.kvc_attn_decode(C.byref(kc), C.byref(vc), T, B, Hkv, Hq, query, 0.1, None, None, 0, out, 2, ws, ws_bytes,
                                               status, None), "kvc_attn_decode")
            else:
                _lib.check(lib.kvc_attn_decode_static(C.byref(kc), C.byref(vc), T, B, Hkv, Hq, query, 0.1, None, None, 0, out, 2,
                                                      status, None), "kvc_attn_decode_static")
        status, ws = ops.new_status("cuda"), ops.attn_workspace(B, Hq, 2, "cuda")
        torch.cuda.synchronize()
        call(kc, vc, query.data_ptr(), out.data_ptr(), codes.data_ptr(), status.data_ptr(), ws.data_ptr(), ws.numel())
        torch.cuda.synchronize()
        result = codes if entry == "decode" else out
        want, zeros = result.cpu(), torch.zeros_like(ws, device="cpu")
        query_host, status_host = query.cpu(), status.cpu()
        got = []
        for _ in range(2):                               # each time a context of its own
            with _Context() as ctx:
                again = []
                for (tensors, spec, n, biggest) in host:
                    p = [ctx.put(t) for t in tensors]
                    meta = _lib.QMeta(p[4], p[5], tensors[4].element_size(), spec.tok_div, spec.sj, spec.sb, spec.sh, spec.sc)
                    again.append(_lib.Cache(p[0], n, p[1], p[2], p[3], meta, biggest, 0))
                r, s = ctx.put(torch.zeros_like(want)), ctx.put(status_host)
                call(again[0], again[1], ctx.put(query_host), r, r, s, ctx.put(zeros), zeros.numel())
                got.append(ctx.get(r, want))
                assert int(ctx.get(s, status_host)) == 0
        call(kc, vc, query.data_ptr(), out.zero_().data_ptr(), codes.zero_().data_ptr(), status.data_ptr(), ws.data_ptr(), ws.numel())
        torch.cuda.synchronize()                         # and the first context is served as before
        got.append(result.cpu())
        q.put("ok" if all(torch.equal(g, want) for g in got) and int(status) == 0 else "wrong output")
    except Exception as e:                               # the parent prints it
        q.put(repr(e))


@pytest.mark.parametrize("entry", ["decode", "attn", "static"])
def test_calls_in_a_second_context_of_the_device(entry):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    p = ctx.Process(target=_second_context, args=(entry, q))
    p.start()
    result = q.get(timeout=180)
    p.join(timeout=60)
    assert result == "ok", result
