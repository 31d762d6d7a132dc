"""Grouped attention over more steps than the device has workers, where vectors are decoded by pairs or symbol by symbol: bad vector starts, bytes that are no
code, staging waits that run out, streams off 16 bytes, an unknown block bound and books without the count of lone windows."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

SCALING = 0.25 / math.sqrt(128)
KW = [dict(), dict(splits=1, workspace=False)]            # partial results and the merge; teams


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops as _ops
    return _ops


def _shape():
    """Columns of so many steps that every worker of the device takes three (five workers on an SM, steps of 128 tokens)."""
    B, H = 16, 4
    return 128 * (3 * 5 * torch.cuda.get_device_properties(0).multi_processor_count // (B * H) + 1), B, H


# symbol frequencies, and the way that the book's windows lead to
BOOKS = {"pairs": [1.0] * 8, "lagging": [2.0 ** -abs(i - 7) for i in range(15)], "singles": [1.0] * 100,
         "no_branch": [2.0 ** -i for i in range(8)] + [2.0 ** -i for i in range(9, 14)]}


class _Cache:
    def __init__(self, ops, kind, is_k, g):
        self.ops = ops
        T, B, H = _shape()
        p = torch.tensor(BOOKS[kind], dtype=torch.float64, device="cuda")
        edges = (p / p.sum()).cumsum(0)
        codes = torch.searchsorted(edges, torch.rand(T * B * H * 128, dtype=torch.float64, device="cuda", generator=g)).clamp_(max=len(p) - 1).to(torch.uint8).view(T, B, H, 128)
        if kind == "no_branch":                            # codes of 1, 2, 3, .. bits, the one of 9 bits taken away
            tree = ops.build_codebook(torch.tensor([2 ** (14 - i) if i < 14 else 0 for i in range(256)], dtype=torch.int64, device="cuda")).ref_decode_tensor()
            nodes = tree.view(-1, 3)
            leaf = [i for i in range(len(nodes)) if nodes[i, 0] == 1 and nodes[i, 1] == 8][0]
            for node in nodes:
                if not node[0]:
                    for side in (1, 2):
                        if node[side] == leaf:
                            node[side] = 0xff
            self.book = ops.book_from_tree(tree.cuda())
            codes = torch.where(codes >= 8, codes + 1, codes)
        else:
            self.book = ops.build_codebook(torch.bincount(codes.flatten().int(), minlength=256))
        lone = self.book.host()[32:36].view(torch.int32).item()
        assert lone >> 16 == 0x4b56 and ((lone & 0xffff) > 100) == (kind == "singles"), (kind, hex(lone))
        self.spec = ops.qspec(ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN, False, B, H, 128, 64)
        units = self.spec.units(T, B, H, 128)
        self.mi = torch.randint(-20, 20, (units,), device="cuda", generator=g).to(torch.int16)
        self.sc = (0.002 + 0.03 * torch.rand(units, device="cuda", generator=g)).half()
        bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
        self.bi, self.ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz // 2, dtype=torch.int16, device="cuda")
        self.enc = torch.empty(2 * n, dtype=torch.uint8, device="cuda")
        total, st = ops.encode(codes, is_k, self.book.encode_table(), self.bi, self.ti, self.enc)
        self.size, self.largest = total.tolist()
        assert ops.read_status(st) == 0

    def arg(self, enc=None, book=None, largest=None):
        return self.ops.make_cache(self.enc if enc is None else enc, self.bi, self.ti, book or self.book, self.mi, self.sc, self.spec, self.size,
                                   self.largest if largest is None else largest)


@pytest.fixture(scope="module", params=[("pairs", "lagging"), ("lagging", "pairs"), ("singles", "no_branch"), ("no_branch", "singles")], ids="-".join)
def caches(request, ops):
    g = torch.Generator(device="cuda").manual_seed(7)
    return request.param, _Cache(ops, request.param[0], True, g), _Cache(ops, request.param[1], False, g)


def _call(ops, k, v, G, kw, fatal=True):
    T, B, H = _shape()
    q = torch.randn(B, H * G, 128, device="cuda", generator=torch.Generator(device="cuda").manual_seed(G)).half()
    out, st = ops.attn_decode(k, v, T, B, H, q, SCALING, **kw)
    return out, ops.read_status(st, raise_on_fatal=fatal)


@pytest.mark.parametrize("kw", KW)
@pytest.mark.parametrize("G", [2, 4, 8])
def test_bad_vector_starts_and_bytes(ops, caches, G, kw):
    """They are flagged, everything else comes out as before, and the call after them is right."""
    (kk, vk), k, v = caches
    clean, st = _call(ops, k.arg(), v.arg(), G, kw)
    assert st == 0
    B = _shape()[1]

    def flagged():
        out, st = _call(ops, k.arg(), v.arg(), G, kw, fatal=False)
        assert st & 0x80 and torch.isfinite(out).all()
        same = [torch.equal(out.view(B, -1)[b], clean.view(B, -1)[b]) for b in range(B)]
        assert sum(same) >= B - 1                          # (a block is one sequence's)

    for c, kind in ((k, kk), (v, vk)):
        ti, enc = c.ti.clone(), c.enc.clone()
        try:
            bits = (c.largest + 40) << 3                   # past the largest block; 16 bits without a sign
            c.ti[64 * 11 + 9] = bits - 65536 if bits >= 32768 else bits
            flagged()
            c.ti.copy_(ti)
            if kind == "no_branch":                        # (of the other books any bits are codes)
                at, n = c.bi.view(torch.int32).view(-1, 2)[200].tolist()
                c.enc[at:at + (n & 0xffff)] = torch.randint(0, 256, (n & 0xffff,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)).to(torch.uint8)
                flagged()
        finally:
            c.ti.copy_(ti)
            c.enc.copy_(enc)
    out, st = _call(ops, k.arg(), v.arg(), G, kw)
    assert st == 0 and torch.equal(out, clean)


@pytest.mark.parametrize("kw", KW)
@pytest.mark.parametrize("G", [2, 4, 8])
def test_staging_waits_run_out(ops, caches, G, kw):
    _, k, v = caches
    T, B, H = _shape()
    clean, st = _call(ops, k.arg(), v.arg(), G, kw)
    assert st == 0
    ws = ops.attn_workspace(B, H * G, ops.attn_splits(T, B, H), "cuda")
    held = dict(workspace=ws) if not kw else kw
    try:
        ops.attn_debug(wait_limit=8, starve=True)
        out, st = _call(ops, k.arg(), v.arg(), G, held, fatal=False)
        assert st & 0x400
    finally:
        ops.attn_debug()
    assert int(ws[:256].view(torch.int32).abs().sum()) == 0          # the scheduling counters were left zeroed
    out, st = _call(ops, k.arg(), v.arg(), G, held)
    assert st == 0 and torch.equal(out, clean)


@pytest.mark.parametrize("kw", KW)
@pytest.mark.parametrize("G", [2, 4, 8])
def test_streams_off_16_bytes_and_an_unknown_bound(ops, caches, G, kw):
    _, k, v = caches
    clean, st = _call(ops, k.arg(), v.arg(), G, kw)
    assert st == 0
    off = []
    for c in (k, v):
        enc = torch.zeros(c.size + 64, dtype=torch.uint8, device="cuda")
        enc[3:3 + c.size] = c.enc[:c.size]
        off.append(enc)
    out, st = _call(ops, k.arg(enc=off[0][3:]), v.arg(enc=off[1][3:]), G, kw)
    assert st == 0 and torch.equal(out, clean)
    # larger slots, fewer workers: another cut of the columns.  (1e-3 of the largest output, as for the attention everywhere)
    out, st = _call(ops, k.arg(largest=0), v.arg(largest=0), G, kw)
    assert st == 0 and float((out.double() - clean.double()).abs().max() / clean.double().abs().max()) <= 1e-3


@pytest.mark.parametrize("word", [0, -1, 0x12345678])
@pytest.mark.parametrize("G", [2, 4, 8])
def test_books_without_the_count_of_lone_windows(ops, caches, G, word):
    """Blobs from before the header had it hold anything there."""
    _, k, v = caches
    clean, st = _call(ops, k.arg(), v.arg(), G, {})
    assert st == 0
    old = []
    for c in (k, v):
        blob = c.book.blob.clone()
        blob[32:36].view(torch.int32)[0] = word
        old.append(type(c.book)(blob))
    out, st = _call(ops, k.arg(book=old[0]), v.arg(book=old[1]), G, {})
    assert st == 0 and torch.equal(out, clean)
