"""The packed arguments of a decode step's and a store's calls have the layout of the structures in the header (CPU)."""
import ctypes as C
import os
import re

import torch

from kvcomp_b200 import _lib, ops
from kvcomp_b200.cache.kvcomp_encode import KVCompCtx
from kvcomp_b200.utils.compute import QuantMode
from kvcomp_b200.utils.config import KVCompCacheConfig, KVCompCacheConfigStatic

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_packed_layouts_match_the_structures():
    assert C.sizeof(_lib.Cache) == 104
    assert _lib.ATTN_ARGS.size == 2 * C.sizeof(_lib.Cache) + 12 * 8 + 8
    assert _lib.KV_STORE_ARGS.size == 11 * 8
    values = list(range(1, 31))
    blob = _lib.ATTN_ARGS.pack(*values, *range(31, 43), 0.5, 7)
    k, v = (_lib.Cache.from_buffer_copy(blob, i * 104) for i in range(2))
    for c, first in ((k, 1), (v, 16)):
        got = [c.encoded, c.encoded_bytes, c.block_info, c.thread_info, c.book, c.q.min_int, c.q.scale, c.q.min_bytes, c.q.tok_div,
               c.q.sj, c.q.sb, c.q.sh, c.q.sc, c.max_block_bytes, c.reserved]
        assert got == list(range(first, first + 15))


def test_packed_store_matches_the_structure():
    """29 words, six numbers of 32 bits, a float and the number of entries."""
    assert _lib.STORE_ARGS.size == 29 * 8 + 8 * 4
    blob = _lib.STORE_ARGS.pack(*range(29), *range(6), 0.5, 0)
    assert int.from_bytes(blob[28 * 8:29 * 8], "little") == 28 and int.from_bytes(blob[29 * 8 + 20:29 * 8 + 24], "little") == 5


STORE_FIELDS = ("x cos_ sin_ cos_batch_stride B H x_tokens T D block codes min_int scale scratch scratch_bytes book enc_codes enc_T base_offset block_info "
                "thread_info encoded encoded_capacity rest rest_rows kept kept_rows report enc_table mode batch_shared heads is_k build min_bytes rel n_entries").split()


def _header_fields(struct):
    """[(name, letter of the struct module)] of a structure in the header."""
    text = open(os.path.join(REPO, "include", "kvcomp_b200.h")).read()
    body = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    body = re.search(r"typedef struct \{([^}]*)\} %s;" % struct, body).group(1)
    fields = []
    for decl in filter(None, (d.strip() for d in body.split(";"))):
        kind, names = re.match(r"(?:const )?(\w+)\s*(.*)", decl, re.S).groups()
        for name in names.split(","):
            pointer = "*" in name
            assert pointer == ("*" in names)
            fields.append((name.strip(" *\n"), "q" if pointer else {"int64_t": "q", "int32_t": "i", "float": "f"}[kind]))
    return fields


def test_packed_store_has_the_headers_fields():
    """The header's fields, in its order, with their sizes: 29 words, six numbers of 32 bits, a float and the number of the encode table's entries."""
    fields = _header_fields("kvc_store_args")
    assert [name for name, _ in fields] == STORE_FIELDS
    letters = re.sub(r"(\d+)(\w)", lambda m: int(m.group(1)) * m.group(2), _lib.STORE_ARGS.format.lstrip("<"))
    assert "".join(letter for _, letter in fields) == letters

    class Args(C.Structure):                                 # as the compiler lays it out
        _fields_ = [(name, {"q": C.c_int64, "i": C.c_int32, "f": C.c_float}[letter]) for name, letter in fields]
    assert C.sizeof(Args) == _lib.STORE_ARGS.size
    a = Args.from_buffer_copy(_lib.STORE_ARGS.pack(*range(35), 0.5, 36))
    assert [getattr(a, name) for name in STORE_FIELDS] == [*range(35), 0.5, 36]


def test_what_a_store_packs(monkeypatch):
    """ops.encode_now and a context's first store, by the names of the structure's fields."""
    packed = []
    monkeypatch.setattr(ops, "_cuda", lambda t, dtype, name: t)
    monkeypatch.setattr(ops, "wait", lambda device: None)
    monkeypatch.setattr(ops.Reports, "place", staticmethod(lambda: (0, 4096)))
    monkeypatch.setattr(ops.Reports, "read", staticmethod(lambda i: [64, 64, 0, 0]))
    monkeypatch.setattr(ops, "store_at", lambda device, words, ints, rel, n_entries=0: packed.append(dict(zip(STORE_FIELDS, [*words, *ints, rel, n_entries]))))
    codes, table, buf = torch.zeros(64, 2, 3, 128, dtype=torch.uint8), torch.zeros(8 * 20, dtype=torch.uint8), torch.zeros(8192, dtype=torch.uint8)
    bi, ti = torch.zeros(48, dtype=torch.uint8), torch.zeros(768, dtype=torch.uint8)
    ops.encode_now(codes, True, table, bi, ti, buf, 77)
    a = packed.pop()
    assert (a["enc_codes"], a["enc_table"], a["n_entries"], a["block_info"], a["thread_info"], a["encoded"], a["encoded_capacity"], a["report"]) == \
        (codes.data_ptr(), table.data_ptr(), 20, bi.data_ptr(), ti.data_ptr(), buf.data_ptr(), 8192, 4096)
    assert (a["T"], a["enc_T"], a["base_offset"], a["B"] * a["H"], a["is_k"], a["build"], a["rest_rows"], a["kept_rows"], a["book"]) == (0, 64, 77, 6, 1, 0, 0, 0, 0)
    KVCompCacheConfigStatic.config = KVCompCacheConfig("synthetic", QuantMode("ChannelQuant"), QuantMode("TokenQuant"), 64, 64, 32, 32, 0.05, 0.1)
    try:
        ctx, x = KVCompCtx(True, 2, 3, 128, 0.05, batch_shared=False, min_dtype=torch.int16, keep_dequantised=True), torch.zeros(2, 3, 200, 128, dtype=torch.float16)
        cos, sin = torch.ones(1, 200, 128, dtype=torch.float16), torch.zeros(1, 200, 128, dtype=torch.float16)
        begun = ctx.begin_heads(x, cos, sin)
    finally:
        KVCompCacheConfigStatic.config = None
    a = packed.pop()
    assert (a["x"], a["cos_"], a["sin_"], a["cos_batch_stride"], a["B"], a["H"], a["x_tokens"], a["T"], a["D"], a["block"]) == \
        (x.data_ptr(), cos.data_ptr(), sin.data_ptr(), 0, 2, 3, 200, 192, 128, 64)
    assert (a["codes"], a["min_int"], a["scale"], a["book"], a["enc_codes"], a["enc_T"], a["base_offset"]) == \
        (begun.pend.data_ptr(), ctx._mi.at, ctx._sc.at, begun.book.blob.data_ptr(), begun.pend.data_ptr(), 192, 0)
    assert (a["block_info"], a["thread_info"], a["encoded"], a["encoded_capacity"]) == (ctx._bi.at, ctx._ti.at, ctx._enc.at, 192 * 6 * 128)
    assert (a["rest"], a["rest_rows"], a["kept"], a["kept_rows"]) == (begun.buf.data_ptr() + 192 * 6 * 256, 8, begun.buf.data_ptr(), 192)
    assert (a["mode"], a["batch_shared"], a["heads"], a["is_k"], a["build"], a["min_bytes"], a["rel"], a["n_entries"], a["enc_table"]) == \
        (_lib.MODE_CHANNEL, False, True, True, True, 2, 0.05, 0, 0)
