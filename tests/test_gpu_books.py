"""Books by the heap of 32-bit and of 64-bit frequencies, their decode tables, and books from a caller's tree whatever its shape."""
import random

import numpy as np
import pytest
import torch

from oracle import kvc_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops as _ops
    return _ops


def _tables(ops, book):
    b = book.host().numpy()
    enc = b[ops.BOOK_OFF_ENC:ops.BOOK_OFF_ENC + 2048].copy().view("<u4").reshape(256, 2)
    off = ops.BOOK_OFF_REFTREE + 1536
    return enc, b[off:off + 2048].copy().view("<u4"), b[off + 2048:off + 2048 + 16384].copy().view("<u4")


def _lut(tree):
    """The decode table bit by bit from the wide tree (lo 16 bits: child 0, or LEAF; hi 16 bits: child 1, or the symbol)."""
    out = np.zeros(4096, np.uint32)
    for w in range(4096):
        syms = n = used = 0
        idx = -1
        for pos in range(12):
            bit = w >> (11 - pos) & 1
            ch = bit if idx == -1 else int(tree[idx]) >> (16 * bit) & 0xffff
            if ch >= 512:
                idx = -2
                break
            node = int(tree[ch])
            if node & 0xffff == LEAF:
                syms |= (node >> 16) << (8 * n)
                n, used, idx = n + 1, pos + 1, -1
                if n == 3:
                    break
            else:
                idx = ch
        out[w] = (syms << 8 | n << 6 | used if n else (NONE if idx < 0 else idx) << 8) & 0xffffffff
    return out


LEAF, NONE = 0xffff, 0xfffe


def _counts(kind, n, rng):
    syms = sorted(rng.sample(range(256), n))
    h = np.zeros(256, np.int64)
    for i, s in enumerate(syms):
        h[s] = {"ties": 5, "few": rng.randint(1, 3), "bell": 1 + int(1e9 * np.exp(-((i - n / 2) / (n / 6 + 1)) ** 2)), "any": rng.randint(1, 1 << 40),
                "steep": 1 << min(i, 50)}[kind]
    return h


@pytest.mark.parametrize("kind", ["ties", "few", "bell", "any", "steep"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 12, 22, 31, 32, 33, 47, 62, 63, 64, 65, 66, 128, 256])
def test_codes_and_tables(ops, kind, n):
    rng = random.Random(n)
    for _ in range(1 if kind == "ties" else 3):
        h = _counts(kind, n, rng)
        book = ops.build_codebook(torch.from_numpy(h).cuda())
        enc, tree, lut = _tables(ops, book)
        want, count = orc.gen_codes(h)
        assert count == n == book.header()["n_symbols"]
        if int(want["length"].max()) > 32:
            continue                                         # flagged; such a book cannot be used
        assert np.array_equal(enc[:, 0], want["code"]) and np.array_equal(enc[:, 1], want["length"])
        if n < 256 and not book.header()["flags"]:
            assert np.array_equal(lut, _lut(tree))


def _walk(t):
    """{symbol: (code, length)} of a reference-format tensor, the last leaf counting, and whether the walk ended by itself."""
    n, out, stack, guard = len(t) // 3, {}, [(1, 1, 1), (0, 0, 1)], 0
    while stack and guard < 2048:
        guard += 1
        nd, code, length = stack.pop()
        if nd >= n:
            continue
        if t[3 * nd]:
            out[int(t[3 * nd + 1])] = (code & 0xffffffff, length)
            continue
        for c, bit in ((int(t[3 * nd + 2]), 1), (int(t[3 * nd + 1]), 0)):
            if c != 0xff and len(stack) < 510:
                stack.append((c, (code << 1 | bit) & (1 << 40) - 1, length + 1))
    return out


def test_books_from_trees(ops):
    """Trees of books, and tensors that no book has: unreachable nodes, missing and out-of-range children, shared children, a symbol at two leaves, roots as
    children, loops that no leaf leaves."""
    rng = random.Random(5)
    for n in (2, 3, 12, 22, 60, 100, 127):
        for change in ("none", "missing", "beyond", "shared", "twice", "root", "unreachable"):
            enc, _ = orc.gen_codes(_counts("few", n, rng))
            t = orc.ref_decode_tree(enc).copy()
            nodes = len(t) // 3
            inner = [i for i in range(nodes) if not t[3 * i]]
            leaves = [i for i in range(nodes) if t[3 * i]]
            i, j = (rng.choice(inner) if inner else None), rng.choice(leaves)
            if change == "missing" and i is not None:
                t[3 * i + 1] = 0xff
            elif change == "beyond" and i is not None:
                t[3 * i + 2] = min(254, nodes + 3)
            elif change == "shared" and i is not None and i < j:
                t[3 * i + 2] = j
            elif change == "twice":
                t[3 * j + 1] = t[3 * j + 2] = t[3 * rng.choice(leaves) + 1]
            elif change == "root" and i is not None and i < 2:
                continue                                     # (a root that leads to itself ends by the walk's bound)
            elif change == "root" and i is not None:
                t[3 * i + 1] = 0xff
                t[3 * i + 2] = rng.choice(leaves)
            elif change == "unreachable" and nodes < 250:
                t = np.concatenate([t, np.array([0, nodes + 1, nodes, 0, nodes, nodes + 2, 1, 250, 250], np.uint8)])      # a loop with a leaf
            want = _walk(t)
            if max(length for _, length in want.values()) > 32:
                continue
            book = ops.book_from_tree(torch.from_numpy(t).cuda())
            got, tree, lut = _tables(ops, book)
            assert {s: (int(got[s, 0]), int(got[s, 1])) for s in range(256) if got[s, 1]} == want, (n, change)
            h = book.header()
            assert (h["n_symbols"], h["min_sym"], h["max_sym"], h["max_len"]) == (len(want), min(want), max(want), max(x for _, x in want.values())), (n, change)
            assert np.array_equal(lut, _lut(tree)), (n, change)
