"""KVCompCtx: the compressed store of one layer's K or V (models/cache/kvcomp_encode.py:15-326).

Same constructor, methods and bookkeeping as the reference class, with the work moved into the CUDA
library: the quantiser is one kernel instead of ~8 torch ops, histogram and codebook are built on the
device, and the stream grows inside pre-reserved arenas instead of torch.cat on every store
(kvcomp_encode.py:129-133).  Beyond the reference: ChannelQuant / VectorQuant for K, per-sequence
units, any batch size in the fused kernels, and `cache()` for the one-pass decode attention.

Tokens are quantised in whole blocks of the configured block size, exactly where the reference cuts
(utils/compute.py:44-72), and encoded in whole Huffman blocks (64 tokens for K, 128 for V).  When a V
block size is not a multiple of 128 (the reference's CUDA path forbids that, kvcomp_encode.py:52-54; its
model path allows it), up to 127 quantised tokens wait as plain codes for their vector to fill.
"""
from typing import NamedTuple

import torch

from .. import ops
from .._lib import KvcError
from ..utils.compute import QuantMode, cut_len, cut_tensor_ctx_len_0
from ..utils.config import KVCompCacheConfigStatic

_MODE = {QuantMode.BlockQuant: ops.MODE_BLOCK, QuantMode.ChannelQuant: ops.MODE_CHANNEL,
         QuantMode.TokenQuant: ops.MODE_TOKEN, QuantMode.VectorQuant: ops.MODE_VECTOR}


class _Arena:
    """A 1-D device buffer that grows geometrically; `n` elements are in use.  Its memory is a tensor of its own or a part of one that several
    arenas share (a context's first store makes one allocation for four of them)."""

    def __init__(self, dtype):
        self.dtype, self.size, self.n = dtype, dtype.itemsize, 0
        self._mem, self._off, self._cap, self._buf = None, 0, 0, None

    def __getstate__(self):                  # a copy makes the view of its own memory anew
        state = self.__dict__.copy()
        if state["_buf"] is not state["_mem"]:
            state["_buf"] = None
        return state

    @property
    def buf(self):
        if self._buf is None and self._mem is not None:
            self._buf = self._mem[self._off:self._off + self._cap * self.size].view(self.dtype)
        return self._buf

    @buf.setter
    def buf(self, t):
        self._mem, self._off, self._cap, self._buf = t, 0, 0 if t is None else t.numel(), t

    @property
    def at(self):
        """Address of the first element."""
        return self._mem.data_ptr() + self._off

    def need(self, extra):
        """Elements to allocate for `extra` more."""
        return max(self.n + extra, int(self._cap * 1.5), 1024)

    def share(self, mem, off, cap):
        """Lie in bytes off .. of `mem`, which nothing else uses."""
        self._mem, self._off, self._cap, self._buf = mem, off, cap, None

    def address(self, extra, device):
        """Where the next `extra` elements go."""
        if self._mem is None or self._cap < self.n + extra:
            new = torch.empty(self.need(extra), dtype=self.dtype, device=device)
            if self.n:
                new[:self.n] = self.buf[:self.n]
            self.buf = new
        return self.at + self.n * self.size

    def reserve(self, extra, device):
        """The next `extra` elements."""
        self.address(extra, device)
        return self.buf[self.n:self.n + extra]

    def used(self):
        """What is in use; None while nothing is, whether there is memory or not."""
        return self.buf[:self.n] if self.n else None


class _RecentRows:
    """The rows behind the compressed stream, fp16 [r, B, H, D], kept in place in one buffer:

        [ kept | recent )      kept:   dequantised values of quantised tokens that a reader still wants as rows
                               recent: the uncompressed recent window (the reference's `buffer`)

    New rows are written behind the recent ones; when the front of the window is compressed its rows are
    overwritten with their dequantised values and join the kept ones (or are given up), so that both parts
    always form one contiguous range and nothing is concatenated at a decode step (the reference's
    torch.cat, models/cache/kvcomp_encode.py:80, copies the whole window, some ten megabytes per tensor and
    layer, at every store).  The rows move to the front only when the end of the buffer is reached."""

    def __init__(self):
        self.buf, self.q, self.lo, self.hi = None, 0, 0, 0

    def __len__(self):                      # recent rows
        return self.hi - self.lo

    @property
    def kept(self):
        return self.lo - self.q

    def view(self):
        return None if self.buf is None else self.buf[self.lo:self.hi]

    def rows_from_kept(self, k):
        """The last k kept rows followed by the recent ones; earlier kept rows are given up."""
        self.q = self.lo - k
        if self.q == self.hi:
            self.q = self.lo = self.hi = 0
            return None
        return self.buf[self.q:self.hi]

    def consume(self, n):
        """The first n recent rows were compressed: their places now belong to the kept rows."""
        self.lo += n

    def reserve(self, t, room, shape, dtype, device):
        """Room for t more rows; returns the rows' place [t, B, H, D] without making them live (commit does)."""
        held = self.hi - self.q
        if self.buf is None or self.hi + t > self.buf.shape[0]:
            if self.buf is not None and held + t <= self.buf.shape[0] and self.q >= held:
                self.buf[:held] = self.buf[self.q:self.hi]          # the two ranges do not overlap
            else:
                new = torch.empty((held + t + room,) + tuple(shape), dtype=dtype, device=device)
                if held:
                    new[:held] = self.buf[self.q:self.hi]
                self.buf = new
            self.lo, self.hi, self.q = self.lo - self.q, held, 0
        return self.buf[self.hi:self.hi + t]

    def commit(self, t):
        self.hi += t

    def append(self, rows, room):
        """Add rows [t, B, H, D]; `room`: rows to leave space for beyond what is needed now."""
        t = rows.shape[0]
        self.reserve(t, room, rows.shape[1:], rows.dtype, rows.device)[:] = rows
        self.commit(t)

    def restart(self, n_old, n_kept, n_recent, buf):
        """Start over in `buf` with the last n_old kept rows (copied), n_kept more and n_recent recent ones (the caller's,
        in their places behind them)."""
        if n_old:
            buf[:n_old] = self.buf[self.lo - n_old:self.lo]
        if n_old + n_kept + n_recent:
            self.buf = buf
        self.q, self.lo, self.hi = 0, n_old + n_kept, n_old + n_kept + n_recent

    def rebuild(self, kept, recent, room):
        """Start over with the given kept rows and recent rows (either may be None)."""
        parts = [p for p in (kept, recent) if p is not None and p.shape[0]]
        nk = 0 if kept is None else kept.shape[0]
        if not parts:
            self.q = self.lo = self.hi = 0
            return
        n = sum(p.shape[0] for p in parts)
        self.buf = torch.empty((n + room,) + tuple(parts[0].shape[1:]), dtype=parts[0].dtype, device=parts[0].device)
        torch.cat(parts, dim=0, out=self.buf[:n])
        self.q, self.lo, self.hi = 0, nk, n

    def set(self, rows):
        self.buf, self.q, self.lo, self.hi = rows, 0, 0, (0 if rows is None else rows.shape[0])


class _Begun(NamedTuple):
    """A store that is on its way: what _finish needs of _launch."""
    slot: int                # of ops.Reports
    book: object             # the book that it encodes with, built by it where the context has none
    pend: object             # codes: `old` rows that waited for their block, then the new ones; None: nobody needs them
    old: int
    part: object             # those of pend that are encoded, n_enc rows
    n_enc: int
    stream_room: int         # bytes for the stream, and the most that it can take
    cap: int
    n_units: int
    n: int                   # tokens that are compressed
    t: int                   # new tokens
    over: bool               # the window starts over in buf: n_old kept rows, k more, n_rest recent ones
    k: int
    n_old: int
    buf: object
    n_rest: int
    put_rest: object         # None: the rest has been written
    blocks: int              # of the stream


class KVCompCtx:
    _cache_arg = _cache_q = None             # (of a copy)
    _given = False                           # a caller has set the window

    def __getstate__(self):                  # the argument structure holds addresses: a copy makes its own
        state = self.__dict__.copy()
        state.pop("_cache_arg", None)
        state.pop("_cache_q", None)
        return state

    def __init__(self, is_k, batch_size, head_num, head_dim, quant_scale_rel,
                 encode_codebook_path=None, decode_codebook_path=None, batch_shared=None, min_dtype=None,
                 keep_dequantised=False):
        """batch_shared / min_dtype: None takes the configuration's quant_per_sequence / wide_min_ints, and
        where those are None too the reference's CUDA-path conventions (units span the batch, int8 min_ints).
        keep_dequantised: keep the fp16 values of freshly quantised tokens until trim_dequantised() drops
        them, so that a decode loop can hand the tokens behind the fused kernel's range over without decoding."""
        cfg = KVCompCacheConfigStatic.config
        assert cfg is not None, "KVCompCacheConfigStatic.config is None"
        assert head_dim == 128, "head_dim must be equal to K_VEC_LEN and V_VEC_LEN for cuda kernel implementation"
        self.is_k = is_k
        self.batch_size, self.head_num, self.head_dim = batch_size, head_num, head_dim
        self.quant_scale_rel = quant_scale_rel
        self.quant_mode = cfg.k_quant_mode if is_k else cfg.v_quant_mode
        self.block_size = cfg.k_block_size if is_k else cfg.v_block_size
        self.recent_size = cfg.k_recent_size if is_k else cfg.v_recent_size
        if batch_shared is None:
            per_seq = getattr(cfg, "quant_per_sequence", None)
            batch_shared = True if per_seq is None else not per_seq
        if min_dtype is None:
            wide = getattr(cfg, "wide_min_ints", None)
            min_dtype = torch.int16 if wide else torch.int8
        self.batch_shared, self.min_dtype = bool(batch_shared), min_dtype
        self.cut_block = self.block_size                     # tokens are quantised where the reference cuts
        if is_k:
            assert self.block_size % 64 == 0, "for K, block size must be divisible by VEC_PER_BLK"
            assert self.quant_mode in _MODE
            self.enc_block = 64
        else:
            assert self.quant_mode in (QuantMode.TokenQuant, QuantMode.VectorQuant, QuantMode.BlockQuant), \
                "V units must not depend on the channel"
            self.enc_block = 128                             # whole 128-token vectors
        if self.quant_mode in (QuantMode.BlockQuant, QuantMode.ChannelQuant) and not is_k:
            assert self.block_size % 128 == 0 or 128 % self.block_size == 0
        self.spec = ops.qspec(_MODE[self.quant_mode], self.batch_shared, batch_size, head_num, head_dim,
                              self.block_size)
        self.ctx_len = 0
        self.compressed_ctx_len = 0              # quantised tokens
        self.encoded_ctx_len = 0                 # of those, the tokens in the stream (whole Huffman blocks)
        self._pending = None                     # codes of quantised tokens whose Huffman block is not full yet
        self.keep_dequantised = keep_dequantised
        self.device = None
        self._recent = _RecentRows()             # uncompressed recent tokens, fp16 [r, B, H, D] (self.buffer)
        self.book = None
        self.max_block_bytes = 0
        self._enc = _Arena(torch.uint8)
        self._bi = _Arena(torch.uint8)
        self._ti = _Arena(torch.int16)
        self._mi = _Arena(self.min_dtype)
        self._sc = _Arena(torch.float16)
        self._cache_arg = self._cache_q = None   # _argument()'s structure

    # ---- views with the reference's attribute names --------------------------------------------
    @property
    def buffer(self):
        return self._recent.view()

    @buffer.setter
    def buffer(self, rows):
        self._recent.set(rows)
        self._given = True                                   # the window may have any shape now

    @property
    def encoded_data(self):
        return self._enc.used()

    @property
    def block_infos(self):
        return self._bi.used()

    @property
    def thread_infos(self):
        u = self._ti.used()
        return None if u is None else u.view(torch.uint8)

    def _unit_shape(self):
        s = self.spec
        B, H, D = self.batch_size, self.head_num, self.head_dim
        nb = 1 if (s.sb == 0) else B
        nh = 1 if (s.sh == 0) else H
        nc = 1 if (s.sc == 0) else D
        per_blk = self.block_size // s.tok_div if s.tok_div <= self.block_size else 1
        return (-1, per_blk, nb, nh, nc)

    @property
    def quant_min_ints(self):
        u = self._mi.used()
        return None if u is None else u.view(*self._unit_shape())

    @property
    def quant_scales(self):
        u = self._sc.used()
        return None if u is None else u.view(*self._unit_shape())

    @property
    def encode_codebook(self):
        return None if self.book is None else self.book.encode_table()

    @property
    def decode_codebook(self):
        return None if self.book is None else self.book.ref_decode_tensor().to(self.device)

    @property
    def shape(self):
        return torch.Size([self.compressed_ctx_len, self.batch_size, self.head_num, self.head_dim])

    # ---- store ------------------------------------------------------------------------------------
    def _room(self):
        return self.recent_size // 2 + self.cut_block          # rows to spare when the window's buffer has to grow

    def recent_place(self, t, device):
        """Where the next t tokens would lie in the recent window, fp16 [t, B, H, D], when storing them compresses
        nothing (the usual decode step), else None.  A caller that can produce the rows there (the rotation and
        transposition kernel) does so and calls recent_commit(t) instead of store(rows)."""
        if self.device is None:
            self.device = device
        if self.device != device or cut_len(len(self._recent) + t, self.cut_block, self.recent_size) // self.cut_block * self.cut_block:
            return None
        return self._recent.reserve(t, self._room(), (self.batch_size, self.head_num, self.head_dim), torch.float16, device)

    def recent_address(self, t, device):
        """recent_place() as an address, for a caller that has check_new() look at the tokens before it writes them there."""
        if self.device is None:
            self.device = device
        r = self._recent
        if self.device != device or self._cut(r.hi - r.lo, t):
            return None
        if r.buf is None or r.hi + t > r.buf.shape[0]:
            r.reserve(t, self._room(), (self.batch_size, self.head_num, self.head_dim), torch.float16, device)
        return self._row_address(r.hi)

    def _row_address(self, i):
        """Address of row i of the window's buffer."""
        b = self._recent.buf
        if b.dtype is not torch.float16 or not b.is_contiguous() or not b.is_cuda:
            ops._cuda(b, torch.float16, "buffer")
        return b.data_ptr() + i * (2 * self.batch_size * self.head_num * self.head_dim)

    def check_new(self, shape):
        """Raise unless new tokens of this shape [B, H, t, D] are rows of the window: their places are sized by it."""
        B, H, _, D = shape
        if B != self.batch_size or H != self.head_num or D != self.head_dim or \
                (self._given and self._recent.buf.shape[1:] != (B, H, D)):
            raise KvcError("new tokens %s for a cache of %d sequences, %d heads, dimension %d and a window %s" % (
                tuple(shape), self.batch_size, self.head_num, self.head_dim, tuple(self._recent.buf.shape)))

    def recent_commit(self, t):
        self._recent.commit(t)
        self.ctx_len += t

    def _check(self, cache):
        assert cache.dtype == torch.float16, "cache must be float16"
        assert cache.shape[1] == self.batch_size, "batch size mismatch"
        assert cache.shape[2] == self.head_num, "head num mismatch"
        assert cache.shape[3] == self.head_dim, "head dim mismatch"
        if self.device is None:
            self.device = cache.device
        assert self.device == cache.device, "device mismatch"

    def _cut(self, live, t):
        """How many of the first tokens of (recent window + t new tokens) are compressed."""
        # utils/compute.py:59-72.  With recent_size = 0 and a ragged length the reference's slice clips to the length and
        # its .view then fails (kvcomp_encode.py:83); here the ragged rest simply stays in the window.
        return min(cut_len(live + t, self.cut_block, self.recent_size), live + t) // self.cut_block * self.cut_block

    def store_heads(self, x, cos=None, sin=None):
        """store() of new tokens as a model's projections leave them, [B, H, t, D], rotated with cos / sin where they
        are given.  A prompt into an empty window is quantised from where it lies."""
        return self._finish(self.begin_heads(x, cos, sin))

    def begin_heads(self, x, cos=None, sin=None, keep_codes=True):
        """store_heads() up to its wait: what finish() takes.  keep_codes = False: the caller has no use for the codes, and their memory
        is the next launch's where nothing else needs them."""
        B, H, t, D = x.shape
        live, mode = len(self._recent), _MODE[self.quant_mode]
        n = self._cut(live, t)
        if live or n == 0 or x.data_ptr() % 16 or not ops.quantize_heads_fits(mode, self.batch_shared, n, B, H, D, self.block_size) \
                or (cos is not None and mode != ops.MODE_CHANNEL):
            return self._begin(ops.rope_store(x, cos, sin), keep_codes)
        cos, sin, stride = ops._rotation(ops._cuda(x, torch.float16, "x"), cos, sin)
        if cos is not None and (cos.data_ptr() | sin.data_ptr()) % 16:
            return self._begin(ops.rope_store(x, cos, sin), keep_codes)
        self._check(x.permute(2, 0, 1, 3))
        return self._launch(x, n, 0, t - n, t, t, None, cos, sin, stride, keep_codes)

    def store(self, cache):
        """Append tokens [t, B, H, D]; whole blocks beyond the recent window are quantised and encoded.
        Returns the uint8 codes of the newly compressed tokens as [n_blocks, block, B, H, D] (or None)."""
        return self._finish(self._begin(cache))

    def _begin(self, cache, keep_codes=True):
        self._check(cache)
        live, t = len(self._recent), cache.shape[0]
        n = self._cut(live, t)
        if n == 0:
            self._recent.append(cache, self._room())          # the usual decode step: the new rows, nothing else moves
            self.ctx_len += t
            return None
        if live == 0:
            x, rest = cache[:n].contiguous(), cache[n:]       # a prefill: compressed from where it lies
        elif n <= live:
            x, rest = self._recent.view()[:n].clone(), cache  # the window's front
        else:
            x, rest = torch.cat([self._recent.view(), cache[:n - live]], dim=0), cache[n - live:]
        return self._launch(x, n, live, rest.shape[0], t, 0, lambda place: place.copy_(rest), keep_codes=keep_codes)

    def _launch(self, x, n, live, n_rest, t, x_tokens, put_rest, cos=None, sin=None, stride=0, keep_codes=True):
        """Launch the compression of the first n tokens of (the `live` rows of the window + t new tokens): x as rows, or (x_tokens > 0) as a
        prompt's heads.  put_rest(place) writes the n_rest last of the new tokens as rows; the heads' own are written by the call.
        Nothing counts before _finish: any step here may fail (an allocation), and the device may refuse the tokens."""
        # quantise, book, encode and the rows are launched by one call; one copy brings back what the kernels report
        # (a prompt of 333 tokens, K and V: a call, a wait and a copy for each kernel 637 us, one report per tensor 409;
        # one call per tensor and one wait for both 261)
        shape, dev = (self.batch_size, self.head_num, self.head_dim), self.device
        B, H, D = shape
        mode, build = _MODE[self.quant_mode], self.book is None
        book = ops.new_book(dev) if build else self.book
        old = 0 if self._pending is None else self._pending.shape[0]
        pend = torch.empty((old + n,) + shape, dtype=torch.uint8, device=dev)
        if old:
            pend[:old] = self._pending
        n_enc = (old + n) // self.enc_block * self.enc_block
        part = pend if n_enc == old + n else pend[:n_enc]
        stream_room, cap = self._encode_room(part) if n_enc else (0, 0)
        blocks = n_enc * B * H * D // 8192
        n_units = self.spec.units(n, B, H, D)
        scratch = torch.empty(ops._lib.load().kvc_store_scratch(mode, self.batch_shared, n, B, H, self.block_size, n_enc, self.is_k), dtype=torch.uint8, device=dev)
        # Where the window starts over, the rest of the new tokens is written before the wait: a caller's tensors are then read
        # when the store returns, whichever stream they belong to.
        over, k, n_old, buf, at_kept, at_rest = live == 0 or n > live, 0, 0, None, 0, 0
        if over:
            if self.keep_dequantised:
                k = min(n, max(self.KEEP_ROWS // self.cut_block, 1) * self.cut_block)    # a long prefill keeps its last rows only
                n_old = self._recent.kept if k == n else 0
            if n_old + k + n_rest:
                buf = torch.empty((n_old + k + n_rest + self._room(),) + shape, dtype=torch.float16, device=dev)
                at_kept = buf.data_ptr() + n_old * (2 * B * H * D)
                at_rest = at_kept + k * (2 * B * H * D)
        if not x_tokens:
            ops._cuda(x, torch.float16, "x")
            if mode in (ops.MODE_BLOCK, ops.MODE_CHANNEL) and n % self.block_size:
                raise KvcError("T=%d is not a multiple of block=%d" % (n, self.block_size))
        if self._bi._mem is None and self._ti._mem is None and self._mi._mem is None and self._sc._mem is None:
            parts, size = ((self._bi, blocks * 8), (self._ti, blocks * 64), (self._mi, n_units), (self._sc, n_units)), 0
            for a, m in parts:
                size += (a.need(m) * a.size + 255) // 256 * 256
            mem, at = torch.empty(size, dtype=torch.uint8, device=dev), 0
            for a, m in parts:
                cap = a.need(m)
                a.share(mem, at, cap)
                at += (cap * a.size + 255) // 256 * 256
        slot, report = ops.Reports.place()
        try:
            ops.store_at(dev, (x.data_ptr(), 0 if cos is None else cos.data_ptr(), 0 if sin is None else sin.data_ptr(), stride, B, H, x_tokens, n, D, self.block_size,
                               pend.data_ptr() + old * (B * H * D), self._mi.address(n_units, dev), self._sc.address(n_units, dev), scratch.data_ptr(), scratch.numel(),
                               book.blob.data_ptr(), pend.data_ptr(), n_enc, self._enc.n, self._bi.address(blocks * 8, dev), self._ti.address(blocks * 64, dev),
                               self._enc.address(stream_room, dev), stream_room, at_rest, n_rest if x_tokens and over else 0, at_kept, k, report, 0),
                         (mode, self.batch_shared, x_tokens > 0, self.is_k, build, self._mi.size), self.quant_scale_rel)
            if over and n_rest and not x_tokens:
                put_rest(buf[n_old + k:n_old + k + n_rest])
        except BaseException:                                 # nothing that is on its way may arrive in the place later
            ops.wait(dev)
            raise
        # A book built from these very codes lacks none of them and the room is for the longest stream: with all of them in the stream and the kept rows
        # written, nothing reads the codes again.  (Keys' and values' on their way together would else be held at the same time.)
        if not keep_codes and build and over and n_enc == old + n:
            pend = part = None
        if over:
            put_rest = None                                   # (it holds the new tokens' rows, all of them)
        return _Begun(slot, book, pend, old, part, n_enc, stream_room, cap, n_units, n, t, over, k, n_old, buf, n_rest, put_rest, blocks)

    def held(self, begun):
        """Bytes that a begun store keeps until _finish: its codes, and the window that another one takes the place of."""
        window = self._recent.buf if begun.over else None
        return (0 if begun.pend is None else begun.pend.numel()) + (0 if window is None else window.numel() * window.element_size())

    def _finish(self, begun, waited=False):
        """The rest of a begun store: waits for it (waited: the caller has), then it counts.  A store that the device refuses does not
        count: the context is as it was, its book too."""
        if begun is None:
            return None
        slot, book, pend, old, part, n_enc, stream_room, cap, n_units, n, t, over, k, n_old, buf, n_rest, put_rest, blocks = begun
        if not waited:
            ops.wait(self.device)
        words, room, codes = ops.Reports.read(slot), self._room(), pend[old:] if old and pend is not None else pend
        flags = ops.check_flags(words[2], what="quantize")
        if flags & ops._lib.FLAG_MIN_OVERFLOW:
            # int8 is the reference's CUDA path, which wraps silently (kvcomp_encode.py:97); its model path
            # keeps min_ints in floating point (utils/compute.py:89).  Wrapped values dequantise wrongly.
            if self.min_dtype == torch.int16:
                raise KvcError("a min_int does not fit 16 bits: the data lies too far from zero for its range")
            import warnings
            warnings.warn("a min_int wrapped in int8 as in the reference's CUDA path; set wide_min_ints to keep it")
        if n_enc and not words[3] & (ops._lib.FLAG_SYMBOL_MISSING | (ops._lib.FLAG_STREAM_FULL if stream_room != cap else 0)):
            ops.check_flags(words[3], what="entropy_encode")  # (the two are seen to below)
        self.book = book
        self.ctx_len += t
        # the window: the compressed rows leave it, or stay as dequantised rows for a reader of the rows behind
        # the fused kernel's range (tail_from); the rest of the new tokens joins the recent rows
        if not over:
            if self.keep_dequantised:
                mi = self._mi.buf[self._mi.n:self._mi.n + n_units]
                sc = self._sc.buf[self._sc.n:self._sc.n + n_units]
                ops.dequant(codes, mi, sc, self.spec, out=self._recent.view()[:n])     # in place of the rows themselves
                self._recent.consume(n)
            else:
                self._recent.consume(n)
                self._recent.rows_from_kept(0)
            if n_rest:
                put_rest(self._recent.reserve(n_rest, room, codes.shape[1:], torch.float16, self.device))
                self._recent.commit(n_rest)
        else:
            self._recent.restart(n_old, k, n_rest, buf)
        self._mi.n += n_units
        self._sc.n += n_units
        self.compressed_ctx_len += n
        if n_enc:
            if not self._encode_finish(part, blocks, stream_room, cap, words):
                # A symbol the frozen book has no code for.  The reference drops such symbols silently
                # (kernels.cu:197-205: a table entry of length 0 adds no bits), which corrupts the stream.
                # Here the book is rebuilt over everything stored so far plus every reachable code, and the
                # cache is re-encoded once; this cannot happen again for this context.
                self._rebook(part)
            self.encoded_ctx_len += n_enc
        self._pending = pend[n_enc:].contiguous() if pend is not None and pend.shape[0] > n_enc else None
        return None if codes is None else codes.view(-1, self.block_size, self.batch_size, self.head_num, self.head_dim)

    def _encode_room(self, codes):
        """Bytes to reserve for the stream of `codes` [T, B, H, D]: (a first guess, the most it can take)."""
        # The reference reserves one byte per symbol (numel) for every store (kernels.cu:903); the stream
        # needs a fraction of that, so room is reserved from the density seen so far (8 bits per symbol at
        # first) with a quarter on top, and the store is repeated with the full reserve in the rare case
        # that the encoder reports the room as exceeded.
        cap = codes.numel()
        seen = self.encoded_ctx_len * self.batch_size * self.head_num * self.head_dim
        return (cap if seen == 0 else min(cap, int(1.25 * self._enc.n / seen * codes.numel()) + 4096)), cap

    def _encode_launch(self, codes, room, report):
        """Encode `codes` into the arenas behind what they hold; nothing counts before _encode_finish."""
        bsz, tsz, _, _ = ops.buffer_sizes(codes.shape[0], self.batch_size * self.head_num * self.head_dim, self.is_k)
        ops.encode(codes, self.is_k, self.book.encode_table(), self._bi.reserve(bsz, self.device),
                   self._ti.reserve(tsz // 2, self.device), self._enc.reserve(room, self.device),
                   base_offset=self._enc.n, total=report.total, status=report.enc_status)

    def _encode_finish(self, codes, blocks, room, cap, words):
        """The launched stream of `blocks` blocks joins the arenas.  False if the book lacks a symbol."""
        if words[3] & ops._lib.FLAG_STREAM_FULL and room != cap:
            self.stream_retries = getattr(self, "stream_retries", 0) + 1
            report = ops.Report(self.device)
            self._encode_launch(codes, cap, report)
            words = report.read()
        if words[3] & ops._lib.FLAG_SYMBOL_MISSING:
            return False
        ops.check_flags(words[3], what="entropy_encode")
        self._enc.n += words[0]
        self._bi.n += blocks * 8
        self._ti.n += blocks * 64
        self.max_block_bytes = max(self.max_block_bytes, words[1])
        return True

    def _encode(self, codes):
        """Append the stream of `codes` [T, B, H, D] to the arenas.  False if the book lacks a symbol."""
        room, cap = self._encode_room(codes)
        report = ops.Report(self.device)
        self._encode_launch(codes, room, report)
        return self._encode_finish(codes, codes.numel() // 8192, room, cap, report.read())

    def _rebook(self, new_codes):
        old = None
        if self.encoded_ctx_len:
            old, st = ops.decode(self._enc.used(), self._bi.used(), self._ti.used(), self.book,
                                 self.encoded_ctx_len, self.batch_size, self.head_num, self.is_k,
                                 max_block=self.max_block_bytes)
            ops.read_status(st, what="entropy_decode")
        hist = ops.histogram(new_codes.view(-1))
        if old is not None:
            hist = ops.histogram(old.view(-1), hist)
        reach = min(255, int(1.0 / self.quant_scale_rel) + 3)      # codes are 0 .. about 1/rel + 1
        hist[:reach + 1] += 1
        self.book = ops.build_codebook(hist)
        self._enc.n = self._bi.n = self._ti.n = 0
        self.max_block_bytes = 0
        self.rebooks = getattr(self, "rebooks", 0) + 1
        for part in (old, new_codes):
            if part is not None and not self._encode(part):
                raise KvcError("a code outside 0..%d appeared; the quantiser settings cannot produce it" % reach)

    def build_codebook(self, tensors):
        """Freeze the codebook from sample tensors before the first store (kvcomp_encode.py:282-306)."""
        assert len(tensors) > 0, "tensors must not be empty"
        hist = None
        for cache in tensors:
            self._check(cache)
            blocked = cache.shape[0] // self.block_size * self.block_size
            if blocked == 0:
                continue
            x = cache[:blocked].contiguous()
            if hist is None:
                hist = torch.zeros(256, dtype=torch.int64, device=self.device)
            mi = torch.empty(self.spec.units(blocked, self.batch_size, self.head_num, self.head_dim),
                             dtype=self.min_dtype, device=self.device)
            ops.quantize(x, _MODE[self.quant_mode], self.block_size, self.quant_scale_rel, self.batch_shared,
                         min_dtype=self.min_dtype, hist=hist, min_int=mi)
        if hist is None:
            raise KvcError("build_codebook: no whole block in the sample tensors")
        self.book = ops.build_codebook(hist)
        hd = self.book.header()
        assert hd["min_sym"] == 0, "shift must be 0"

    # ---- read back --------------------------------------------------------------------------------
    def _require(self):
        assert self.compressed_ctx_len > 0 and self.book is not None, "nothing has been compressed yet"

    def get_decode_quant_ints(self):
        """Decoded uint8 codes [n_blocks, block, B, H, D] and the kernel time in ms."""
        self._require()
        out = None
        with ops.TimedCall.on(self.device) as call:
            if self.encoded_ctx_len:
                out, _ = ops.decode(self._enc.used(), self._bi.used(), self._ti.used(), self.book,
                                    self.encoded_ctx_len, self.batch_size, self.head_num, self.is_k,
                                    status=call.status, max_block=self.max_block_bytes)
            ms = call.end("entropy_decode")
        if self._pending is not None:
            out = self._pending if out is None else torch.cat([out, self._pending], dim=0)
        return out.view(-1, self.block_size, self.batch_size, self.head_num, self.head_dim), ms

    def _values(self, rows):
        """An fp16 tensor of `rows` tokens whose first compressed_ctx_len are the dequantised values, decoded and
        dequantised by one kernel (plain codes that wait for their Huffman block: dequantised behind them), and its
        time in ms."""
        self._require()
        n, shape = self.encoded_ctx_len, (self.batch_size, self.head_num, self.head_dim)
        with ops.TimedCall.on(self.device) as call:
            x = torch.empty((rows,) + shape, dtype=torch.float16, device=self.device)
            if n:
                ops.decode_values(self._argument(), n, *shape[:2], self.is_k, x[:n], status=call.status)
            if self._pending is not None:
                first = n // self.spec.tok_div * self.spec.sj                # unit of the first waiting token
                ops.dequant(self._pending, self._mi.used()[first:], self._sc.used()[first:], self.spec, out=x[n:self.compressed_ctx_len])
            return x, call.end("entropy_decode")

    def get_only_compressed(self):
        """Dequantised compressed part [T, B, H, D] and the time of decode + dequantisation in ms."""
        return self._values(self.compressed_ctx_len)

    def get(self):
        """Whole cache [ctx_len, B, H, D]: dequantised compressed part followed by the recent window."""
        if self.compressed_ctx_len == 0:
            return self.buffer, 0.0
        recent = self.buffer
        live = 0 if recent is None else recent.shape[0]
        x, t = self._values(self.compressed_ctx_len + live)
        if live:
            x[self.compressed_ctx_len:] = recent
        return x, t

    def cache(self):
        """The kvc_cache argument of the fused kernels over the encoded_ctx_len tokens of the stream (valid
        until the next store).  A structure of the caller's own."""
        return ops.copy_cache(self._argument())

    def _argument(self):
        """The same for a launch made right away: this context's one structure, every field that a store can change
        filled in again at each call (0.8 us; a new structure 2 us)."""
        assert self.encoded_ctx_len > 0 and self.book is not None, "nothing has been encoded yet"
        c = self._cache_arg
        if c is None:
            # (from addresses: as tensors, the parts of a shared allocation took 10 us of a cache's first get() or mat_vec_mul())
            s = self.spec
            c = self._cache_arg = ops.Cache(self._enc.at, self._enc.n, self._bi.at, self._ti.at, self.book.blob.data_ptr(),
                                            ops.QMeta(self._mi.at, self._sc.at, self._mi.size, s.tok_div, s.sj, s.sb, s.sh, s.sc), self.max_block_bytes, 0)
            self._cache_q = c.q
            return c
        c.encoded, c.encoded_bytes, c.max_block_bytes = self._enc.at, self._enc.n, self.max_block_bytes
        c.block_info, c.thread_info, c.book = self._bi.at, self._ti.at, self.book.blob.data_ptr()
        self._cache_q.min_int, self._cache_q.scale = self._mi.at, self._sc.at
        return c

    def _fields(self):
        """cache()'s contents in the order of the structure, for a launch made right away."""
        assert self.encoded_ctx_len > 0 and self.book is not None, "nothing has been encoded yet"
        s, e = self.spec, self._enc
        return (e.at, e.n, self._bi.at, self._ti.at, self.book.blob.data_ptr(), self._mi.at, self._sc.at, self._mi.size, s.tok_div, s.sj, s.sb, s.sh, s.sc, self.max_block_bytes, 0)

    def mat_vec_mul(self, B):
        """K: scores [batch, heads, ctx] = q . K^T; V: [1, batch, heads, 128] = P . V over the compressed
        tokens (kvcomp_encode.py:209-280).  Returns (tensor, ms)."""
        self._require()
        if self._pending is not None:
            raise KvcError("mat_vec_mul: %d quantised tokens are not in the stream yet (V block sizes that are "
                           "no multiple of 128 leave such a rest)" % self._pending.shape[0])
        assert B.dtype == torch.float16, "B must be float16"
        assert len(B.shape) == 3, "B must be 3D tensor"
        assert B.shape[0] == self.batch_size, "batch size mismatch"
        hq = B.shape[1]
        assert hq % self.head_num == 0, "head num mismatch"
        if self.is_k:
            assert B.shape[2] == self.head_dim, "head dim mismatch"
        else:
            assert B.shape[2] == self.compressed_ctx_len, "ctx len mismatch"
        with ops.TimedCall.on(self.device) as call:
            if self.is_k:
                C, _ = ops.fused_qk(self._argument(), self.compressed_ctx_len, self.batch_size, self.head_num, B, status=call.status)
            else:
                part, _ = ops.fused_pv(self._argument(), self.compressed_ctx_len, self.batch_size, self.head_num, B, status=call.status)
                C = ops.pv_sum(part)
            return C, call.end("mat_vec_mul")

    def save(self, path):
        """Write this cache to a file (kvcomp_b200.cache.storage describes the format)."""
        from .storage import save_ctx
        return save_ctx(self, path)

    @staticmethod
    def load(path, device="cuda"):
        from .storage import load_ctx
        return load_ctx(path, device)

    def get_cr(self):
        """Compression ratio with the reference's accounting (kvcomp_encode.py:317-326)."""
        compressed = (self._bi.n + self._ti.n * 2 + self._enc.n + self._mi.n * self._mi.used().element_size() +
                      self._sc.n * 2)
        pending = 0 if self._pending is None else self._pending.numel()
        original = 2 * self.batch_size * self.compressed_ctx_len * self.head_num * self.head_dim
        return original / (compressed + pending)

    # ---- the tokens behind the fused kernel's range ---------------------------------------------------
    KEEP_ROWS = 512       # dequantised rows a long store keeps at most (tail_from decodes when it needs more)

    def tail_from(self, T):
        """fp16 [n, B, H, D]: the quantised tokens from index T on (dequantised) followed by the recent
        window, as one range of the window's buffer.  Dequantised rows before T are given up."""
        need = max(0, self.compressed_ctx_len - T)
        if need > self._recent.kept:
            # not kept (keep_dequantised off, a cache read from a file, a prefill longer than KEEP_ROWS whose
            # other tensor lags far behind): decode the stream once, keep the rows from T on
            x, _ = self.get_only_compressed()
            kept = x[T:].contiguous()
            if not self.keep_dequantised:
                return kept if not len(self._recent) else torch.cat([kept, self._recent.view()], dim=0)
            self._recent.rebuild(kept, self._recent.view(), self._room())
        return self._recent.rows_from_kept(need)

    def tail_at(self, T):
        """tail_from(T) as (address, rows); None when the rows have to be made first."""
        r = self._recent
        need = max(0, self.compressed_ctx_len - T)
        if need > r.lo - r.q:
            return None
        r.q = r.lo - need
        if r.q == r.hi:
            r.q = r.lo = r.hi = 0
            return 0, 0
        return self._row_address(r.q), r.hi - r.q

    def trim_dequantised(self, T):
        self._recent.rows_from_kept(min(self._recent.kept, max(0, self.compressed_ctx_len - T)))
