"""KVCompCache: the KV-cache object the patched model files construct and call
(models/cache/kvcomp_cache.py:22-38, models/cache/kvcomp_quant.py:14-123; call sites
models/llama.py:279-283,848-852, models/mistral.py:168-171,840-844, models/phi3.py:197-201,916-920).

    cache = KVCompCache(batch_size, head_num, head_dim, layer_num)
    k, v = cache.update(key_states, value_states, layer_idx, {"cos": cos, "sin": sin})   # drop-in
    out = cache.attend(query_states, layer_idx, scaling)                                 # fused path

`update` keeps the reference's contract and returns the reference's values: RoPE is applied to the new
keys inside, the tokens are appended, and the whole cache comes back as fp16 [B, H, T, D] for eager
attention -- compressed blocks dequantised (what the reference's simulated path returns,
kvcomp_quant.py:70-75), recent tokens as they are.  Like that path, quant units never span the batch
(utils/compute.py:138-143) and min_ints are not narrowed to int8, unless the configuration's
quant_per_sequence / wide_min_ints say otherwise.  `append` + `attend` is the path that never
materialises K/V: the tokens go into the compressed store and one kernel computes
softmax(q K^T * scaling) V straight from the streams.
"""
import inspect
import math

import torch

from .. import ops
from .._lib import KvcError
from ..utils.compute import apply_rotary_pos_emb_single, safe_cat
from ..utils.config import KVCompCacheConfigStatic
from .kvcomp_encode import KVCompCtx

try:                                    # transformers 4.50's Cache takes no constructor arguments
    from transformers import Cache as _HFCache
    _BASE = _HFCache if not [p for p in list(inspect.signature(_HFCache.__init__).parameters.values())[1:]
                             if p.default is inspect.Parameter.empty and p.kind in (p.POSITIONAL_ONLY, p.POSITIONAL_OR_KEYWORD)] else object
except Exception:                       # pragma: no cover
    _BASE = object


class KVCompCache(_BASE):
    def __init__(self, batch_size, head_num, head_dim, layer_num):
        if _BASE is not object:
            try:
                super().__init__()
            except Exception:
                pass
        if KVCompCacheConfigStatic.config is None:
            raise ValueError("KVCompCacheConfigStatic.config is not set. Please set it before using KVCompCache.")
        self.batch_size, self.head_num, self.head_dim, self.layer_num = batch_size, head_num, head_dim, layer_num
        self.k_ctx = [None] * layer_num       # created at the first update: the KV head count is only known then
        self.v_ctx = [None] * layer_num
        self.k_plain = [None] * layer_num     # enable_quant = False: plain fp16 concatenation [B, H, T, D]
        self.v_plain = [None] * layer_num
        self.coss = [None] * layer_num
        self.sins = [None] * layer_num
        self._ws = {}
        self._status = {}
        self._last = None

    # ---- appending --------------------------------------------------------------------------------
    def _ctx(self, layer_idx, kv_heads):
        cfg = KVCompCacheConfigStatic.config
        if self.k_ctx[layer_idx] is None:
            kw = dict(batch_shared=getattr(cfg, "quant_per_sequence", None) is False,
                      min_dtype=torch.int8 if getattr(cfg, "wide_min_ints", None) is False else torch.int16,
                      keep_dequantised=True)
            self.k_ctx[layer_idx] = KVCompCtx(True, self.batch_size, kv_heads, self.head_dim, cfg.k_quant_scale_rel, **kw)
            self.v_ctx[layer_idx] = KVCompCtx(False, self.batch_size, kv_heads, self.head_dim, cfg.v_quant_scale_rel, **kw)
        return self.k_ctx[layer_idx], self.v_ctx[layer_idx]

    def append(self, key_states, value_states, layer_idx, cache_kwargs=None):
        """Add new tokens (key/value_states: [B, Hkv, t, D]); keys get RoPE here unless pre-RoPE is on."""
        cfg = KVCompCacheConfigStatic.config
        cos, sin = cache_kwargs["cos"], cache_kwargs["sin"]
        k_stored, begun = False, None
        if cfg.enable_pre_rope:
            self.coss[layer_idx] = safe_cat(self.coss[layer_idx], cos, dim=1)
            self.sins[layer_idx] = safe_cat(self.sins[layer_idx], sin, dim=1)
        elif cfg.enable_quant and key_states.is_cuda and key_states.dtype == torch.float16 and key_states.is_contiguous() \
                and cos.dtype == torch.float16 and key_states.shape[3] % 16 == 0:
            kc0, vc0 = self._ctx(layer_idx, key_states.shape[1])
            t = key_states.shape[2]
            if value_states.is_cuda and value_states.dtype == torch.float16 and value_states.is_contiguous() \
                    and value_states.shape == key_states.shape:
                device = key_states.device
                kplace, vplace = kc0.recent_address(t, device), vc0.recent_address(t, device)
                if kplace is not None and vplace is not None:   # the usual decode step: one launch, straight into both windows
                    if value_states.device != device:
                        raise KvcError("keys on %s, values on %s" % (device, value_states.device))
                    kc0.check_new(key_states.shape)
                    vc0.check_new(key_states.shape)
                    ops.kv_store_at(key_states, value_states, cos, sin, kplace, vplace)
                    kc0.recent_commit(t)
                    vc0.recent_commit(t)
                    return
            place = kc0.recent_place(key_states.shape[2], key_states.device)
            if place is not None:                               # the usual decode step: straight into the recent window
                ops.rope_store(key_states, cos, sin, out=place)
                kc0.recent_commit(key_states.shape[2])
            else:
                begun = kc0.begin_heads(key_states, cos, sin, keep_codes=False)      # rotated with torch's bits
            k_stored = True
        else:
            key_states = apply_rotary_pos_emb_single(key_states, cos, sin)
        if not cfg.enable_quant:
            self.k_plain[layer_idx] = safe_cat(self.k_plain[layer_idx], key_states, dim=2)
            self.v_plain[layer_idx] = safe_cat(self.v_plain[layer_idx], value_states, dim=2)
            return
        kc, vc = self._ctx(layer_idx, key_states.shape[1])
        if not k_stored:
            kc.store(key_states.permute(2, 0, 1, 3).contiguous().half())
        if begun is not None:
            both, begun = self._values_begun(kc, vc, begun, value_states), None      # (no codes of the keys are held from here on)
            if both:
                return
        t = value_states.shape[2]
        plain = self._plain(value_states)
        place = vc.recent_place(t, value_states.device) if plain else None
        if place is not None:                                   # the transposition alone, straight into the window
            ops.rope_store(value_states, None, None, out=place)
            vc.recent_commit(t)
        elif plain and value_states.data_ptr() % 16 == 0:
            vc.store_heads(value_states)
        else:
            vc.store(value_states.permute(2, 0, 1, 3).contiguous().half())

    @staticmethod
    def _plain(x):
        return x.is_cuda and x.dtype == torch.float16 and x.is_contiguous() and x.shape[3] % 16 == 0

    # Bytes that the keys' store may hold while the values' is launched.  A first prompt's holds nothing; a later one's codes and window came on top of
    # all that the values' store takes (2048 tokens of 128 heads behind 2000 others: at its peak 329 MB, 239 one after the other).  One wait for both
    # saves some 35 us whatever the size: 590 and 626 us with 67 MB of codes, 920 and 954 with 134, 1641 and 1669 with 268.
    HELD = 64 << 20

    @staticmethod
    def _values_begun(kc, vc, begun, values):
        """Finish the store of keys that has begun; True if the values' store went with it, behind one wait for both."""
        v_begun = None
        try:
            # (one wait is for one device)
            if KVCompCache._plain(values) and values.data_ptr() % 16 == 0 and values.device == kc.device and kc.held(begun) <= KVCompCache.HELD \
                    and vc.recent_place(values.shape[2], values.device) is None:
                v_begun = vc.begin_heads(values, keep_codes=False)
        finally:
            kc._finish(begun)                                   # waits for both; the values do not count where the keys are refused
        if v_begun is None:
            return False
        vc._finish(v_begun, waited=True)
        return True

    def update(self, key_states, value_states, layer_idx, cache_kwargs=None):
        """The reference's Cache.update: append, then return the whole K and V as [B, Hkv, T, D]."""
        cfg = KVCompCacheConfigStatic.config
        self.append(key_states, value_states, layer_idx, cache_kwargs)
        if not cfg.enable_quant:
            k, v = self.k_plain[layer_idx], self.v_plain[layer_idx]
        else:
            k = self.k_ctx[layer_idx].get()[0].permute(1, 2, 0, 3)
            v = self.v_ctx[layer_idx].get()[0].permute(1, 2, 0, 3)
        if cfg.enable_pre_rope:
            k = apply_rotary_pos_emb_single(k, self.coss[layer_idx], self.sins[layer_idx])
        return k, v

    def get_seq_length(self, layer_idx=0):
        layer_idx = 0 if layer_idx is None else layer_idx
        if not KVCompCacheConfigStatic.config.enable_quant:
            return 0 if self.k_plain[layer_idx] is None else self.k_plain[layer_idx].shape[2]
        return 0 if self.k_ctx[layer_idx] is None else self.k_ctx[layer_idx].ctx_len

    # ---- fused decode attention -------------------------------------------------------------------
    def _tails(self, kc, vc):
        """Length of the range the fused kernel reads from the streams and the fp16 tails behind it.  K and V
        cut their recent windows with different block and window sizes and fill Huffman blocks of
        different length, so either may have quantised tokens beyond that range: their dequantised values
        (kept since they were quantised) go in front of the recent window."""
        T = min(kc.encoded_ctx_len, vc.encoded_ctx_len) // 128 * 128
        return T, kc.tail_from(T), vc.tail_from(T)

    def check(self):
        """Raise if a fused launch since the last check reported a fatal condition (a stream that does not
        decode, a staging wait that ran out).  Synchronises; attend() itself never does."""
        for st in self._status.values():
            flags = ops.read_status(st, what="attend")
            if flags:
                st.zero_()

    def attend(self, query_states, layer_idx, scaling=None):
        """One decode step: query_states [B, Hq, 1, D] (or [B, Hq, D]), already rotated -> attention
        output of the same shape, computed straight from the compressed K and V of the layer; tokens
        that are not in the streams yet (the recent window) are read as fp16 rows by the same kernel.
        With pre-RoPE keys the stored keys are not rotated, every token would need its own rotation of
        the query, and the step goes through the dequantised cache instead (the slow way)."""
        cfg = KVCompCacheConfigStatic.config
        q = query_states
        squeeze = q.dim() == 4
        if squeeze and q.shape[2] != 1:
            raise KvcError("attend handles one query token (decode); use update() for prefill")
        if (squeeze or q.dim() == 3) and cfg.enable_quant and not cfg.enable_pre_rope and q.dtype is torch.float16 and q.is_cuda \
                and q.is_contiguous() and q.shape[-1] == 128 and self.k_ctx[layer_idx] is not None:
            out = self._attend_step(q, self.k_ctx[layer_idx], self.v_ctx[layer_idx], scaling)
            if out is not None:
                return out
        if squeeze:
            q = q[:, :, 0, :]
        q = q.contiguous().half()
        B, Hq, D = q.shape
        scaling = 1.0 / math.sqrt(D) if scaling is None else scaling
        if not cfg.enable_quant or cfg.enable_pre_rope:
            out = self._attend_dense(q, layer_idx, scaling)
            return out.unsqueeze(2) if squeeze else out
        kc, vc = self.k_ctx[layer_idx], self.v_ctx[layer_idx]
        if kc is None:
            raise KvcError("attend before any update")
        T, ktail, vtail = self._tails(kc, vc)
        if T == 0 and ktail is None:
            raise KvcError("empty cache")
        ws, st = self._scratch(q, T, kc.head_num)
        out, _ = ops.attn_decode(kc._argument() if T else None, vc._argument() if T else None, T, B, kc.head_num, q, scaling,
                                 ktail, vtail, splits=0, workspace=ws, status=st)
        return out.unsqueeze(2) if squeeze else out

    def _scratch(self, q, T, kv_heads):
        """Workspace and status word of a launch for q [B, Hq, ...] over T tokens of the streams."""
        B, Hq, device = q.shape[0], q.shape[1], q.device
        last = self._last                                   # (T stays for 64 steps and more)
        if last is not None and last[0] == (device, B, Hq, kv_heads, T):
            return last[1], last[2]
        parts = ops.attn_splits(T, B, kv_heads)             # partial results per head of the balanced split
        ws = self._ws.get((device, B, Hq, parts))
        if ws is None:
            ws = self._ws[(device, B, Hq, parts)] = ops.attn_workspace(B, Hq, parts, device)
        st = self._status.get(device)
        if st is None:
            st = self._status[device] = ops.new_status(device)
        self._last = (device, B, Hq, kv_heads, T), ws, st
        return ws, st

    def _attend_step(self, q, kc, vc, scaling):
        """attend() for a query that lies ready for the kernel, over tails that are in place; else None.  No tensor is
        made but the output, and the launch's arguments are packed at once."""
        T = min(kc.encoded_ctx_len, vc.encoded_ctx_len) // 128 * 128
        ktail, vtail = kc.tail_at(T), vc.tail_at(T)
        if ktail is None or vtail is None or (T == 0 and ktail[1] == 0) or (ktail[1] and not vtail[1]):
            return None
        ws, st = self._scratch(q, T, kc.head_num)
        out = torch.empty(q.shape, dtype=torch.float16, device=q.device)
        ops.attn_decode_at(kc._fields() if T else None, vc._fields() if T else None, T, q.shape[0], kc.head_num, q, out,
                           1.0 / math.sqrt(q.shape[-1]) if scaling is None else float(scaling), ktail[0], vtail[0], ktail[1], ws, st)
        return out

    def _attend_dense(self, q, layer_idx, scaling):
        """softmax(q K^T * scaling) V over the materialised cache: plain fp16 caches (enable_quant off) and
        pre-RoPE caches."""
        cfg = KVCompCacheConfigStatic.config
        if not cfg.enable_quant:
            k, v = self.k_plain[layer_idx], self.v_plain[layer_idx]
        else:
            k = self.k_ctx[layer_idx].get()[0].permute(1, 2, 0, 3)
            v = self.v_ctx[layer_idx].get()[0].permute(1, 2, 0, 3)
        if k is None:
            raise KvcError("attend before any update")
        if cfg.enable_pre_rope:
            k = apply_rotary_pos_emb_single(k, self.coss[layer_idx], self.sins[layer_idx])
        g = q.shape[1] // k.shape[1]
        kf, vf = k.float().repeat_interleave(g, dim=1), v.float().repeat_interleave(g, dim=1)
        w = torch.softmax(torch.einsum("bhd,bhtd->bht", q.float(), kf) * scaling, dim=-1)
        return torch.einsum("bht,bhtd->bhd", w, vf).half()
