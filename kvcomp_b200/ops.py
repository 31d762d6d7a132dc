"""torch-facing wrappers over the C ABI: tensors in, tensors out, launches on the current stream.

PyTorch is only the carrier of device memory and streams here; every computation is a kernel of
libkvcomp_b200.so.  Every function raises when the tensors are not CUDA tensors: there is no CPU path.
"""
import ctypes as C
import functools
import threading
from dataclasses import dataclass

import torch

from . import _lib
from ._lib import (BOOK_BYTES, BOOK_OFF_ENC, BOOK_OFF_REFTREE, MODE_BLOCK, MODE_CHANNEL, MODE_TOKEN,
                   MODE_VECTOR, Cache, KvcError, QMeta)

MODES = {"BlockQuant": MODE_BLOCK, "ChannelQuant": MODE_CHANNEL, "TokenQuant": MODE_TOKEN,
         "VectorQuant": MODE_VECTOR}


# The current device and stream are asked for at every call (a caller may switch either), through the
# interpreter's direct entries where this torch has them: the public context manager and stream object cost
# some ten microseconds per call, as much as the rest of a call's host work.
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_get_device = getattr(torch._C, "_cuda_getDevice", None)
_current_stream = getattr(torch._C, "_cuda_getCurrentStream", None)


def _stream():
    if _raw_stream is not None and _get_device is not None:
        return _raw_stream(_get_device())
    return torch.cuda.current_stream().cuda_stream


class _on:
    """`with _on(device):` makes the tensor's device current for the call, switching only when it is not."""
    __slots__ = ("idx", "prev")

    def __init__(self, device):
        self.idx = device.index if isinstance(device, torch.device) else torch.device(device).index

    def __enter__(self):
        self.prev = _get_device() if _get_device is not None else torch.cuda.current_device()
        if self.idx is not None and self.idx != self.prev:
            torch.cuda.set_device(self.idx)
        return self

    def __exit__(self, *exc):
        if self.idx is not None and self.idx != self.prev:
            torch.cuda.set_device(self.prev)
        return False


def _cuda(t, dtype, name):
    if not isinstance(t, torch.Tensor) or not t.is_cuda:
        raise KvcError("%s must be a CUDA tensor (kvcomp_b200 has no CPU path)" % name)
    if dtype is not None and t.dtype != dtype:
        raise KvcError("%s must be %s, got %s" % (name, dtype, t.dtype))
    if not t.is_contiguous():
        raise KvcError("%s must be contiguous" % name)
    return t


def _p(t):
    return t.data_ptr() if t is not None else None      # a plain number converts faster than a c_void_p object


def new_status(device):
    """A zeroed device status word; kernels OR KVC_FLAG_* bits into it."""
    return torch.zeros(1, dtype=torch.int32, device=device)


def read_status(status, raise_on_fatal=True, what="kvcomp_b200"):
    """Synchronising read of a status word."""
    return check_flags(int(status.item()), raise_on_fatal, what)


def check_flags(v, raise_on_fatal=True, what="kvcomp_b200"):
    """The flags of a status word that is on the host already."""
    if raise_on_fatal and (v & _lib.FATAL_FLAGS):
        raise KvcError("%s: device reported %s" % (what, "|".join(_lib.flag_names(v))))
    return v


class TimedCall:
    """What a call that returns only after the device has finished, with its time and its status, needs: two events and a status
    word.  One per thread and device, kept; the status word is zero between calls.  It lies in pinned memory, where the kernels write it (only
    to report something) and the host reads it: no copy of it stands between the last kernel and the host.
    `with TimedCall.on(device) as call:` begins; the launches and end() belong in the block, so that a call which an exception
    ends is waited for and its flags go with it.
    (Events, a zeroed word and a pageable read-back made anew cost such a call some 20 us, a copy of the word 8.)"""
    __slots__ = ("start", "stop", "status", "flags", "raw", "stream", "device", "open")
    _kept = threading.local()

    def __init__(self, device):
        self.start, self.stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        self.device = device
        with torch.inference_mode(False):                  # a normal tensor, whatever mode the thread's first call runs in:
            self.status = torch.zeros(1, dtype=torch.int32).pin_memory()       # it is written again in calls of either mode
        self.flags = self.status.numpy()
        self.raw = self.stream = None
        self.open = False                                  # launches may be under way that write the status word

    @staticmethod
    def on(device):
        kept = TimedCall._kept.__dict__
        c = kept.get(device)
        if c is None:
            c = kept[device] = TimedCall(device)
        return c

    def _current(self):
        """The device's current stream; the object is made anew only when the stream is another one."""
        if _current_stream is None:
            self.stream = torch.cuda.current_stream(self.device)
            return self.stream
        raw = _current_stream(self.device.index)
        if raw != self.raw:
            self.raw, self.stream = raw, torch.cuda.Stream(stream_id=raw[0], device_index=raw[1], device_type=raw[2])
        return self.stream

    def __enter__(self):
        self.start.record(self._current())
        self.open = True
        return self

    def __exit__(self, *exc):
        if self.open:
            self._clear()
        return False

    def _clear(self):
        """Zero the word behind everything the call has launched."""
        self.stream.synchronize()
        self.flags[0] = 0
        self.open = False

    def end(self, what):
        """Waits; the time since the call began in ms.  Raises on a fatal status."""
        stream = self._current()
        self.stop.record(stream)
        stream.synchronize()
        v = int(self.flags[0])
        self.flags[0] = 0
        self.open = False
        check_flags(v, what=what)
        return self.start.elapsed_time(self.stop)


class Report:
    """What an encoder launched by itself reports -- its byte count and largest block, its status word -- in one zeroed int64[4] laid out as
    a store's (Reports), so that one copy brings all of it to the host."""
    __slots__ = ("words", "total", "enc_status")

    def __init__(self, device):
        self.words = torch.zeros(4, dtype=torch.int64, device=device)
        self.total, self.enc_status = self.words[:2], self.words[3:].view(torch.int32)[:1]

    def read(self):
        """(bytes, largest block, 0, encoder flags); synchronises."""
        return self.words.tolist()


class Reports:
    """Where the reports of a thread's stores arrive: two in pinned memory (a cache's K and V are on their way together), kept per thread.  A
    store takes a place, launches, and reads its words behind a wait."""
    _kept = threading.local()

    def __init__(self):
        with torch.inference_mode(False):
            self.words = torch.zeros(2, 4, dtype=torch.int64).pin_memory()
        self.view, self.next = self.words.numpy(), 0

    @staticmethod
    def place():
        """(index, address) of a place that no store of this thread is using: the stores of one wait are two at most."""
        r = getattr(Reports._kept, "r", None)
        if r is None:
            r = Reports._kept.r = Reports()
        i = r.next
        r.next = 1 - i
        return i, r.words.data_ptr() + 32 * i

    @staticmethod
    def read(i):
        """(bytes, largest block, quantiser flags, encoder flags) of a store that has been waited for."""
        return Reports._kept.r.view[i].tolist()


def wait(device):
    """Wait for the device's current stream."""
    with _on(device):
        _lib.check(_lib.load().kvc_stream_wait(_stream()), "wait")


@dataclass(frozen=True)
class QSpec:
    """Unit layout of a (min_int, scale) pair: unit = (t // tok_div)*sj + b*sb + h*sh + c*sc."""
    mode: int
    batch_shared: bool
    block: int
    tok_div: int
    sj: int
    sb: int
    sh: int
    sc: int

    def units(self, T, B, H, D):
        """Number of units of T tokens."""
        return (T // self.tok_div) * self.sj if self.sj else 0

    def qmeta(self, min_int, scale):
        return QMeta(min_int.data_ptr(), scale.data_ptr(), min_int.element_size(), self.tok_div,
                     self.sj, self.sb, self.sh, self.sc)


@functools.lru_cache(maxsize=256)
def qspec(mode, batch_shared, B, H, D, block):
    lib = _lib.load()
    q = QMeta()
    n = C.c_int64(0)
    T = block if mode in (MODE_BLOCK, MODE_CHANNEL) else 1
    _lib.check(lib.kvc_qmeta_make(mode, int(batch_shared), T, B, H, D, block, C.byref(q), C.byref(n)), "kvc_qmeta_make")
    return QSpec(mode, bool(batch_shared), int(block), q.tok_div, q.sj, q.sb, q.sh, q.sc)


def buffer_sizes(tokens, hidden, is_k):
    out = (C.c_int64 * 4)()
    _lib.check(_lib.load().kvc_buffer_sizes(tokens, hidden, int(is_k), out), "kvc_buffer_sizes")
    return tuple(int(v) for v in out)


def quantize(x, mode, block, rel, batch_shared=True, min_dtype=torch.int8, hist=None, status=None,
             codes=None, min_int=None, scale=None):
    """x: fp16 [T,B,H,D] -> (codes u8 [T,B,H,D], min_int [units], scale fp16 [units], QSpec, status)."""
    lib = _lib.load()
    _cuda(x, torch.float16, "x")
    if x.dim() != 4:
        raise KvcError("x must be [T,B,H,D]")
    T, B, H, D = x.shape
    spec = qspec(mode, batch_shared, B, H, D, block)
    if mode in (MODE_BLOCK, MODE_CHANNEL) and T % block:
        raise KvcError("T=%d is not a multiple of block=%d" % (T, block))
    n = spec.units(T, B, H, D)
    dev = x.device
    codes = torch.empty((T, B, H, D), dtype=torch.uint8, device=dev) if codes is None else _cuda(codes, torch.uint8, "codes")
    min_int = torch.empty(n, dtype=min_dtype, device=dev) if min_int is None else _cuda(min_int, None, "min_int")
    scale = torch.empty(n, dtype=torch.float16, device=dev) if scale is None else _cuda(scale, torch.float16, "scale")
    if min_int.dtype not in (torch.int8, torch.int16) or min_int.numel() < n or scale.numel() < n:
        raise KvcError("min_int must be int8/int16 and hold %d units" % n)
    status = new_status(dev) if status is None else status
    ws_bytes = lib.kvc_quantize_workspace(mode, int(batch_shared), T, B, block)
    ws = torch.empty(max(ws_bytes, 16), dtype=torch.uint8, device=dev)
    if hist is not None:
        _cuda(hist, torch.int64, "hist")
    with _on(dev):
        _lib.check(lib.kvc_quantize(_p(x), T, B, H, D, mode, int(batch_shared), block, float(rel), _p(codes),
                                    _p(min_int), min_int.element_size(), _p(scale), _p(hist), _p(ws), ws.numel(),
                                    _p(status), _stream()), "kvc_quantize")
    return codes, min_int, scale, spec, status


def quant_minmax(x, mode, block, batch_shared=True):
    """Per-unit extremes of x (fp16 [T,B,H,D]) for BlockQuant / TokenQuant units: (min fp16 [units], max
    fp16 [units], QSpec).  First half of the two-call quantiser (kvc_quant_minmax)."""
    lib = _lib.load()
    _cuda(x, torch.float16, "x")
    T, B, H, D = x.shape
    spec = qspec(mode, batch_shared, B, H, D, block)
    n = spec.units(T, B, H, D)
    mn = torch.empty(n, dtype=torch.float16, device=x.device)
    mx = torch.empty(n, dtype=torch.float16, device=x.device)
    ws = torch.empty(max(8 * n, 16), dtype=torch.uint8, device=x.device)
    with _on(x.device):
        _lib.check(lib.kvc_quant_minmax(_p(x), T, B, H, D, mode, int(batch_shared), block, _p(mn), _p(mx), _p(ws),
                                        ws.numel(), _stream()), "kvc_quant_minmax")
    return mn, mx, spec


def quantize_ranged(x, mode, block, rel, mn, mx, batch_shared=True, min_dtype=torch.int8, hist=None, status=None):
    """Second half: quantise x with the given per-unit extremes (the joint ones of all head shards).
    Returns what quantize returns."""
    lib = _lib.load()
    _cuda(x, torch.float16, "x")
    _cuda(mn, torch.float16, "mn")
    _cuda(mx, torch.float16, "mx")
    T, B, H, D = x.shape
    spec = qspec(mode, batch_shared, B, H, D, block)
    n = spec.units(T, B, H, D)
    if mn.numel() != n or mx.numel() != n:
        raise KvcError("extremes must hold %d units" % n)
    dev = x.device
    codes = torch.empty((T, B, H, D), dtype=torch.uint8, device=dev)
    min_int = torch.empty(n, dtype=min_dtype, device=dev)
    scale = torch.empty(n, dtype=torch.float16, device=dev)
    status = new_status(dev) if status is None else status
    ws = torch.empty(max(8 * n, 16), dtype=torch.uint8, device=dev)
    if hist is not None:
        _cuda(hist, torch.int64, "hist")
    with _on(dev):
        _lib.check(lib.kvc_quantize_ranged(_p(x), T, B, H, D, mode, int(batch_shared), block, float(rel), _p(mn), _p(mx),
                                           _p(codes), _p(min_int), min_int.element_size(), _p(scale), _p(hist), _p(ws),
                                           ws.numel(), _p(status), _stream()), "kvc_quantize_ranged")
    return codes, min_int, scale, spec, status


def _rotation(x, cos, sin):
    """cos and sin for x [B, H, t, D], checked, and their stride between sequences (both None: no rotation)."""
    if cos is None:
        return None, None, 0
    B, _, t, D = x.shape
    cos, sin = _cuda(cos.contiguous(), torch.float16, "cos"), _cuda(sin.contiguous(), torch.float16, "sin")
    s = cos.shape
    if s != sin.shape or len(s) != 3 or s[1] != t or s[2] != D or s[0] not in (1, B):
        raise KvcError("cos / sin must be [B, t, D] or [1, t, D], got %s" % (tuple(s),))
    return cos, sin, 0 if s[0] == 1 and B > 1 else t * D


def rope_store(x, cos, sin, out=None, first=0):
    """New keys x fp16 [B, H, t, D] rotated (t * cos + rotate_half(t) * sin in fp16, as torch evaluates it) and
    laid out token-major: fp16 [t, B, H, D].  cos / sin: fp16 [B, t, D] or [1, t, D]; both None: no rotation,
    the transposition alone (new values).  out: where the rows go (a row range of the recent window).
    first: the tokens from this one on, t - first rows."""
    lib = _lib.load()
    _cuda(x, torch.float16, "key_states")
    B, H, x_tokens, D = x.shape
    cos, sin, stride = _rotation(x, cos, sin)
    t = x_tokens - first
    out = torch.empty((t, B, H, D), dtype=torch.float16, device=x.device) if out is None else _cuda(out, torch.float16, "out")
    if tuple(out.shape) != (t, B, H, D):
        raise KvcError("out must be [t, B, H, D] = %s, got %s" % ((t, B, H, D), tuple(out.shape)))
    with _on(x.device):
        _lib.check(lib.kvc_rope_store_rows(_p(x), _p(cos), _p(sin), _p(out), B, H, x_tokens, first, t, D, stride, _stream()), "kvc_rope_store")
    return out


def quantize_heads_fits(mode, batch_shared, T, B, H, D, block):
    """Whether quantize_heads takes T tokens in these units."""
    return bool(_lib.load().kvc_quantize_heads_fits(mode, int(batch_shared), T, B, H, D, block))


def quantize_heads(x, T, cos, sin, mode, block, rel, batch_shared, min_int, scale, hist=None, status=None):
    """The first T tokens of a prompt x fp16 [B, H, t, 128] as its projections leave it, rotated with cos / sin where
    they are given: the codes u8 [T, B, H, 128], min_int and scale that quantize gives for rope_store's rows, without
    the rows.  (For callers of their own: a context's store quantises, builds its book and encodes in one call, store_at.)"""
    lib = _lib.load()
    _cuda(x, torch.float16, "x")
    B, H, t, D = x.shape
    cos, sin, stride = _rotation(x, cos, sin)
    _cuda(min_int, None, "min_int"), _cuda(scale, torch.float16, "scale")
    codes = torch.empty((T, B, H, D), dtype=torch.uint8, device=x.device)
    status = new_status(x.device) if status is None else status
    if hist is not None:
        _cuda(hist, torch.int64, "hist")
    with _on(x.device):
        _lib.check(lib.kvc_quantize_heads(_p(x), _p(cos), _p(sin), stride, B, H, t, T, D, mode, int(batch_shared), block, float(rel),
                                          _p(codes), _p(min_int), min_int.element_size(), _p(scale), _p(hist), _p(status), _stream()),
                   "kvc_quantize_heads")
    return codes


def kv_store(k, v, cos, sin, kout, vout):
    """rope_store for the new keys (rotated) and the new values (not rotated) in one launch: k, v fp16
    [B, H, t, D] -> kout, vout fp16 [t, B, H, D] (row ranges of the recent windows)."""
    lib = _lib.load()
    _cuda(k, torch.float16, "key_states")
    _cuda(v, torch.float16, "value_states")
    B, H, t, D = k.shape
    cos, sin, stride = _rotation(k, cos, sin)
    if tuple(v.shape) != (B, H, t, D) or tuple(kout.shape) != (t, B, H, D) or tuple(vout.shape) != (t, B, H, D):
        raise KvcError("kv_store: k, v must be [B, H, t, D] and kout, vout [t, B, H, D]")
    _cuda(kout, torch.float16, "kout")
    _cuda(vout, torch.float16, "vout")
    with _on(k.device):
        _lib.check(lib.kvc_kv_store(_p(k), _p(v), _p(cos), _p(sin), _p(kout), _p(vout), B, H, t, D, stride, _stream()), "kvc_kv_store")


def kv_store_at(k, v, cos, sin, kaddr, vaddr):
    """kv_store of k and v (CUDA fp16 tensors of one shape, contiguous) to addresses with room for their rows."""
    B, H, t, D = k.shape
    cos, sin, stride = _rotation(k, cos, sin)
    args = _lib.KV_STORE_ARGS.pack(k.data_ptr(), v.data_ptr(), cos.data_ptr(), sin.data_ptr(), kaddr, vaddr, B, H, t, D, stride)
    with _on(k.device):
        _lib.check(_lib.load().kvc_kv_store_packed(args, _stream()), "kvc_kv_store")


def dequant(codes, min_int, scale, spec, out=None):
    lib = _lib.load()
    _cuda(codes, torch.uint8, "codes")
    T, B, H, D = codes.shape
    out = torch.empty((T, B, H, D), dtype=torch.float16, device=codes.device) if out is None else out
    q = spec.qmeta(_cuda(min_int, None, "min_int"), _cuda(scale, torch.float16, "scale"))
    with _on(codes.device):
        _lib.check(lib.kvc_dequant(_p(codes), C.byref(q), T, B, H, D, _p(out), _stream()), "kvc_dequant")
    return out


def histogram(codes, hist=None):
    """hist (int64[256], device) += bincount(codes)."""
    lib = _lib.load()
    _cuda(codes, torch.uint8, "codes")
    hist = torch.zeros(256, dtype=torch.int64, device=codes.device) if hist is None else _cuda(hist, torch.int64, "hist")
    with _on(codes.device):
        _lib.check(lib.kvc_histogram(_p(codes), codes.numel(), _p(hist), _stream()), "kvc_histogram")
    return hist


class Book:
    """A device codebook blob (encode table, reference-format decode tree, decode tables)."""

    def __init__(self, blob):
        self.blob = blob
        self._host = None

    @property
    def device(self):
        return self.blob.device

    def host(self):
        """Synchronising copy of the blob to the host (cached)."""
        if self._host is None:
            self._host = self.blob.cpu()
        return self._host

    def header(self):
        h = self.host()[:32].view(torch.int32).tolist()
        return dict(n_symbols=h[0], min_sym=h[1], max_sym=h[2], max_len=h[3], n_nodes=h[4], flags=h[5], lut_bits=h[6],
                    escape=h[7])

    def encode_table(self):
        """uint8 view of the 256-entry symbol-indexed {u32 code, u32 length} table (device)."""
        return self.blob[BOOK_OFF_ENC:BOOK_OFF_ENC + 2048]

    def ref_encode_tensor(self):
        """(shift, CPU uint8 tensor): the encode tensor of the reference's build_codebook."""
        hd = self.header()
        lo, hi = hd["min_sym"], hd["max_sym"]
        return lo, self.host()[BOOK_OFF_ENC + 8 * lo: BOOK_OFF_ENC + 8 * (hi + 1)].clone()

    def ref_decode_tensor(self):
        """CPU uint8 tensor: the decode tensor of the reference's build_codebook (3-byte nodes)."""
        n = self.header()["n_nodes"]
        return self.host()[BOOK_OFF_REFTREE: BOOK_OFF_REFTREE + 3 * n].clone()


def new_book(device):
    """A book that a store builds."""
    return Book(torch.empty(BOOK_BYTES, dtype=torch.uint8, device=device))


def store_at(device, words, ints, rel, n_entries=0):
    """kvc_store: its arguments' words and ints in the structure's order.  The caller has checked the tensors."""
    with _on(device):
        _lib.check(_lib.load().kvc_store_packed(_lib.STORE_ARGS.pack(*words, *ints, rel, n_entries), _stream()), "store")


def build_codebook(hist):
    lib = _lib.load()
    _cuda(hist, torch.int64, "hist")
    blob = torch.empty(BOOK_BYTES, dtype=torch.uint8, device=hist.device)
    with _on(hist.device):
        _lib.check(lib.kvc_build_codebook(_p(hist), _p(blob), _stream()), "kvc_build_codebook")
    return Book(blob)


def book_from_tree(ref_tree):
    lib = _lib.load()
    _cuda(ref_tree, torch.uint8, "decode_code_book")
    blob = torch.empty(BOOK_BYTES, dtype=torch.uint8, device=ref_tree.device)
    with _on(ref_tree.device):
        _lib.check(lib.kvc_book_from_tree(_p(ref_tree), ref_tree.numel(), _p(blob), _stream()), "kvc_book_from_tree")
    return Book(blob)


def encode(codes, is_k, enc_table, block_info, thread_info, encoded, base_offset=0, status=None, total=None):
    """codes u8 [T,B,H,128] -> writes block_info (u8, 8 B per block), thread_info (2 B per vector) and
    encoded (u8) in place; returns (total, status) where total is a device int64[2]: [0] the byte count
    of this call, [1] the largest block byte count (a running maximum when `total` is passed in again).
    enc_table: device uint8 tensor of {u32 code, u32 length} entries indexed by symbol."""
    lib = _lib.load()
    T, cols = _encode_checks(codes, is_k, enc_table, block_info, thread_info, encoded, base_offset)
    dev = codes.device
    status = new_status(dev) if status is None else status
    total = torch.zeros(2, dtype=torch.int64, device=dev) if total is None else total
    ws = torch.empty(max(lib.kvc_encode_workspace(T, cols, int(is_k)), 16), dtype=torch.uint8, device=dev)
    with _on(dev):
        _lib.check(lib.kvc_encode(_p(codes), T, cols, int(is_k), _p(enc_table), enc_table.numel() // 8,
                                  int(base_offset), _p(block_info), _p(thread_info), _p(encoded),
                                  encoded.numel(), _p(total), _p(ws), ws.numel(), _p(status), _stream()), "kvc_encode")
    return total, status


def _encode_checks(codes, is_k, enc_table, block_info, thread_info, encoded, base_offset):
    """Raise unless the encoder can take these; returns (T, sequences x heads)."""
    _cuda(codes, torch.uint8, "codes")
    T, B, H, D = codes.shape
    if D != 128:
        raise KvcError("head_dim must be 128")
    cols = B * H
    _cuda(enc_table, torch.uint8, "encode_code_book")
    for t, n in ((block_info, "block_infos"), (thread_info, "thread_infos"), (encoded, "encoded_data")):
        _cuda(t, None, n)
    nblk = (T // 64) * cols if is_k else (T // 128) * cols * 2
    if block_info.numel() * block_info.element_size() < nblk * 8 or \
            thread_info.numel() * thread_info.element_size() < nblk * 128:
        raise KvcError("block_infos / thread_infos too small for %d blocks" % nblk)
    if not 0 <= int(base_offset) < 1 << 32:
        raise KvcError("a block's offset has 32 bits, the stream begins at %d" % int(base_offset))
    return T, cols


def encode_now(codes, is_k, enc_table, block_info, thread_info, encoded, base_offset):
    """encode() and a wait; returns (bytes, largest block, 0, status)."""
    T, cols = _encode_checks(codes, is_k, enc_table, block_info, thread_info, encoded, base_offset)
    dev = codes.device
    scratch = torch.empty(_lib.load().kvc_store_scratch(0, 1, 0, 1, cols, 64, T, int(is_k)), dtype=torch.uint8, device=dev)
    slot, report = Reports.place()
    try:
        store_at(dev, (0, 0, 0, 0, 1, cols, 0, 0, 128, 64, 0, 0, 0, scratch.data_ptr(), scratch.numel(), 0, codes.data_ptr(), T, int(base_offset),
                       block_info.data_ptr(), thread_info.data_ptr(), encoded.data_ptr(), encoded.numel(), 0, 0, 0, 0, report, enc_table.data_ptr()),
                 (0, 1, 0, int(is_k), 0, 1), 0.0, enc_table.numel() // 8)
    finally:
        wait(dev)
    return Reports.read(slot)


def decode(encoded, block_info, thread_info, book, T, B, H, is_k, out=None, status=None, max_block=0):
    """Huffman-decode a stream to its uint8 codes [T,B,H,128].  max_block: the stream's largest block in
    bytes as the encoder reported it (0 = unknown); a known bound lets more blocks be at work on an SM."""
    lib = _lib.load()
    _cuda(encoded, torch.uint8, "encoded")
    dev = encoded.device
    out = torch.empty((T, B, H, 128), dtype=torch.uint8, device=dev) if out is None else _cuda(out, torch.uint8, "out")
    status = new_status(dev) if status is None else status
    with _on(dev):
        _lib.check(lib.kvc_decode_bounded(_p(encoded), encoded.numel(), _p(block_info), _p(thread_info), _p(book.blob),
                                          T, B * H, int(is_k), int(max_block), _p(out), _p(status), _stream()), "kvc_decode")
    return out, status


def decode_values(cache, T, B, H, is_k, out, status=None):
    """Huffman-decode a cache's stream of T tokens and dequantise it in the same launch: out fp16 [T,B,H,128], the bits
    of dequant(decode(...)).  Returns the status word."""
    _cuda(out, torch.float16, "out")
    if tuple(out.shape) != (T, B, H, 128):
        raise KvcError("out must be [T,B,H,128] = %s, got %s" % ((T, B, H, 128), tuple(out.shape)))
    status = new_status(out.device) if status is None else status
    with _on(out.device):
        _lib.check(_lib.load().kvc_decode_values(C.byref(cache), T, B, H, int(is_k), _p(out), _p(status), _stream()),
                   "kvc_decode_values")
    return status


def make_cache(encoded, block_info, thread_info, book, min_int, scale, spec, encoded_bytes=None, max_block_bytes=0):
    """The kvc_cache argument of the fused kernels.  The tensors must stay alive during the call."""
    n = encoded.numel() if encoded_bytes is None else int(encoded_bytes)
    return Cache(encoded.data_ptr(), n, block_info.data_ptr(), thread_info.data_ptr(), book.blob.data_ptr(),
                 spec.qmeta(min_int, scale), int(max_block_bytes), 0)


def copy_cache(cache):
    """Another kvc_cache argument with the same contents."""
    return Cache.from_buffer_copy(cache)


def fused_qk(cache, T, B, Hkv, q, out=None, out_dtype=torch.float16, status=None):
    """q fp16 [B,Hq,128] -> raw scores [B,Hq,T]."""
    lib = _lib.load()
    _cuda(q, torch.float16, "q")
    Hq = q.shape[1]
    out = torch.empty((B, Hq, T), dtype=out_dtype, device=q.device) if out is None else _cuda(out, None, "C")
    if out.dtype not in (torch.float16, torch.float32):
        raise KvcError("scores must be fp16 or fp32")
    status = new_status(q.device) if status is None else status
    with _on(q.device):
        _lib.check(lib.kvc_fused_qk(C.byref(cache), T, B, Hkv, Hq, _p(q), _p(out), int(out.dtype == torch.float32),
                                    _p(status), _stream()), "kvc_fused_qk")
    return out, status


def fused_pv(cache, T, B, Hkv, P, out=None, status=None):
    """P fp16 [B,Hq,T] -> per-group partials fp16 [T/128, B, Hq, 128]."""
    lib = _lib.load()
    _cuda(P, torch.float16, "P")
    Hq = P.shape[1]
    out = torch.empty((T // 128, B, Hq, 128), dtype=torch.float16, device=P.device) if out is None else _cuda(out, torch.float16, "C")
    status = new_status(P.device) if status is None else status
    with _on(P.device):
        _lib.check(lib.kvc_fused_pv(C.byref(cache), T, B, Hkv, Hq, _p(P), _p(out), _p(status), _stream()), "kvc_fused_pv")
    return out, status


def pv_sum(part):
    """The groups' partials of fused_pv summed: fp16 [n, B, Hq, 128] -> fp16 [1, B, Hq, 128]."""
    _cuda(part, torch.float16, "part")
    n, B, Hq, _ = part.shape
    out = torch.empty((1, B, Hq, 128), dtype=torch.float16, device=part.device)
    with _on(part.device):
        _lib.check(_lib.load().kvc_pv_sum(_p(part), n, B, Hq, _p(out), _stream()), "kvc_pv_sum")
    return out


def attn_splits(T, B, Hkv):
    return int(_lib.load().kvc_attn_splits(T, B, Hkv, 0))


def attn_workspace(B, Hq, splits, device):
    """Zeroed workspace for attn_decode with up to `splits` splits (reusable across calls)."""
    n = _lib.load().kvc_attn_workspace(B, Hq, splits)
    return torch.zeros(n, dtype=torch.uint8, device=device)


def attn_decode(kcache, vcache, T, B, Hkv, q, scaling, ktail=None, vtail=None, out=None, splits=0,
                workspace=None, status=None):
    """One decode step: q fp16 [B,Hq,128] -> out fp16 [B,Hq,128] over T compressed (+ tail) tokens."""
    lib = _lib.load()
    _cuda(q, torch.float16, "q")
    Hq = q.shape[1]
    dev = q.device
    out = torch.empty((B, Hq, 128), dtype=torch.float16, device=dev) if out is None else _cuda(out, torch.float16, "out")
    status = new_status(dev) if status is None else status
    Tr = 0
    if ktail is not None and ktail.shape[0] > 0:
        _cuda(ktail, torch.float16, "ktail")
        _cuda(vtail, torch.float16, "vtail")
        Tr = ktail.shape[0]
    else:
        ktail = vtail = None
    # splits <= 0: the tiles of all (sequence, KV head) columns are shared evenly among the CTAs that
    # fit the device (attn_splits = partial results per head to leave room for); splits > 0: every
    # column is cut into that many equal parts.
    if workspace is None:
        workspace = attn_workspace(B, Hq, splits if splits > 0 else attn_splits(T, B, Hkv), dev)
    elif workspace is False:        # no workspace at all (splits must be 1): the CTAs take fixed shares of the columns
        workspace = torch.empty(0, dtype=torch.uint8, device=dev)
    with _on(dev):
        _lib.check(lib.kvc_attn_decode(C.byref(kcache) if kcache is not None else None,
                                       C.byref(vcache) if vcache is not None else None, T, B, Hkv, Hq, _p(q), float(scaling),
                                       _p(ktail), _p(vtail), Tr, _p(out), int(splits),
                                       _p(workspace if workspace.numel() else None), workspace.numel(),
                                       _p(status), _stream()), "kvc_attn_decode")
    return out, status


_NO_CACHE = (0,) * 15


def attn_decode_at(kfields, vfields, T, B, Hkv, q, out, scaling, ktail, vtail, Tr, workspace, status):
    """attn_decode with splits = 0 for a caller that makes the call at every step: q and out CUDA fp16 tensors
    [B, Hq, 128] (or [B, Hq, 1, 128]), contiguous; the caches as KVCompCtx._fields() (None while T is 0), the tails as
    addresses."""
    args = _lib.ATTN_ARGS.pack(*(kfields or _NO_CACHE), *(vfields or _NO_CACHE), T, B, Hkv, q.shape[1], q.data_ptr(), ktail, vtail, Tr,
                               out.data_ptr(), workspace.data_ptr(), workspace.numel(), status.data_ptr(), scaling, 0)
    with _on(q.device):
        _lib.check(_lib.load().kvc_attn_decode_packed(args, _stream()), "kvc_attn_decode")


def encode_debug(wait_limit=0, starve=False):
    """Diagnostics of the encoder's bounded waits between blocks (kvc_encode_debug); (0, False) restores the
    defaults."""
    _lib.load().kvc_encode_debug(int(wait_limit), int(bool(starve)))


def decode_debug(wait_limit=0, starve=False):
    """Diagnostics of the decoder's bounded waits for a block's bytes (kvc_decode_debug); (0, False) restores the defaults."""
    _lib.load().kvc_decode_debug(int(wait_limit), int(bool(starve)))


def attn_debug(wait_limit=0, starve=False):
    """Diagnostics of the attention kernel's bounded staging waits (kvc_attn_debug); (0, False) restores
    the defaults."""
    _lib.load().kvc_attn_debug(int(wait_limit), int(bool(starve)))


def attn_decode_static(kcache, vcache, T, B, Hkv, q, scaling, out, ktail=None, vtail=None, splits=0, status=None):
    """attn_decode for callers that must not allocate: the split-KV scratch is the library's built-in
    array, `out` and `status` are the caller's tensors, and this wrapper creates no tensor either.
    Calls that overlap on the GPU share the scratch and race; keep them on one stream."""
    lib = _lib.load()
    _cuda(q, torch.float16, "q")
    _cuda(out, torch.float16, "out")
    if status is None:
        raise KvcError("attn_decode_static: pass a status tensor (ops.new_status) made beforehand")
    Tr = 0
    if ktail is not None and ktail.shape[0] > 0:
        _cuda(ktail, torch.float16, "ktail")
        _cuda(vtail, torch.float16, "vtail")
        Tr = ktail.shape[0]
    else:
        ktail = vtail = None
    with _on(q.device):
        _lib.check(lib.kvc_attn_decode_static(C.byref(kcache), C.byref(vcache), T, B, Hkv, q.shape[1], _p(q),
                                              float(scaling), _p(ktail), _p(vtail), Tr, _p(out), int(splits),
                                              _p(status), _stream()), "kvc_attn_decode_static")
    return out


def k_matvec(k, q, out):
    lib = _lib.load()
    for t, n in ((k, "A"), (q, "B"), (out, "C")):
        _cuda(t, torch.float16, n)
    ctx, bsz, H, D = k.shape
    if bsz != 1 or D != 128:
        raise KvcError("Batch size must be 1 for now")
    with _on(k.device):
        _lib.check(lib.kvc_k_matvec(_p(k), _p(q), _p(out), ctx, H, _stream()), "kvc_k_matvec")
    return out
