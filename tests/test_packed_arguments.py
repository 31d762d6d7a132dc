"""The packed arguments of a decode step's calls have the layout of the structures in the header (CPU)."""
import ctypes as C

from kvcomp_b200 import _lib


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
    """29 words, six numbers of 32 bits, a float and a word that is not used."""
    assert _lib.STORE_ARGS.size == 29 * 8 + 8 * 4
    blob = _lib.STORE_ARGS.pack(*range(29), *range(6), 0.5, 0)
    assert int.from_bytes(blob[28 * 8:29 * 8], "little") == 28 and int.from_bytes(blob[29 * 8 + 20:29 * 8 + 24], "little") == 5
