"""Books from a caller's tree that lacks a branch: some bit patterns belong to no code.  A stream of the symbols that are there decodes without a
flag in every kernel, whatever lies behind a vector's last symbol."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops as _ops
    return _ops


def _book(ops, missing, twice):
    """Codes of 1, 2, 3, .. bits, without that of `missing` bits (twice: its leaf holds the next symbol, which then has two); the symbols."""
    n = 14
    tree = ops.build_codebook(torch.tensor([2 ** (n - i) if i < n else 0 for i in range(256)], dtype=torch.int64, device="cuda")).ref_decode_tensor()
    nodes = tree.view(-1, 3)
    leaf = [i for i in range(len(nodes)) if nodes[i, 0] == 1 and nodes[i, 1] == missing - 1]
    assert len(leaf) == 1
    for node in nodes:
        if not twice and not node[0]:
            for side in (1, 2):
                if node[side] == leaf[0]:
                    node[side] = 0xff
    if twice:
        nodes[leaf[0], 1] = nodes[leaf[0], 2] = missing
    book = ops.book_from_tree(tree.cuda())
    head = book.header()
    assert head["n_symbols"] == n - 1 and head["max_len"] == n - 1 and head["escape"] == 1
    assert int((book.host()[64:64 + 2048].view(torch.int32).view(256, 2)[:, 1] > 0).sum()) == n - 1
    return book, [i for i in range(n) if i != missing - 1]


def _cache(ops, missing, twice, shape, is_k, g):
    T, B, H, _ = shape
    book, symbols = _book(ops, missing, twice)
    p = torch.tensor([2.0 ** -i for i in symbols], device="cuda", dtype=torch.float64)
    edges = (p / p.sum()).cumsum(0)
    at = torch.searchsorted(edges, torch.rand(math.prod(shape), dtype=torch.float64, device="cuda", generator=g)).clamp_(max=len(p) - 1)
    codes = torch.tensor(symbols, device="cuda", dtype=torch.uint8)[at].view(shape)
    spec = ops.qspec(ops.MODE_CHANNEL if is_k else ops.MODE_TOKEN, False, B, H, 128, 64)
    units = spec.units(T, B, H, 128)
    mi = torch.randint(-20, 20, (units,), device="cuda", generator=g).to(torch.int16)
    sc = (0.002 + 0.03 * torch.rand(units, device="cuda", generator=g)).half()
    bsz, tsz, _, n = ops.buffer_sizes(T, B * H * 128, is_k)
    bi, ti = torch.empty(bsz, dtype=torch.uint8, device="cuda"), torch.empty(tsz // 2, dtype=torch.int16, device="cuda")
    enc = torch.empty(2 * n, dtype=torch.uint8, device="cuda")
    total, st = ops.encode(codes, is_k, book.encode_table(), bi, ti, enc)
    size, largest = total.tolist()
    assert ops.read_status(st) == 0
    u = (torch.arange(T, device="cuda") // spec.tok_div)[:, None, None, None] * spec.sj + torch.arange(B, device="cuda")[None, :, None, None] * spec.sb + \
        torch.arange(H, device="cuda")[None, None, :, None] * spec.sh + torch.arange(128, device="cuda")[None, None, None, :] * spec.sc
    return ops.make_cache(enc, bi, ti, book, mi, sc, spec, size, largest), (codes.double() + mi[u].double()) * sc[u].double(), (enc, bi, ti, book, mi, sc)


@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("missing,twice", [(5, False), (9, False), (9, True)])
@pytest.mark.parametrize("long", [False, True])        # a step per worker at most; several
def test_tree_without_a_branch(ops, G, missing, twice, long):
    g = torch.Generator(device="cuda").manual_seed(missing + G)
    B, H = 16, 4
    steps = 4 * 5 * torch.cuda.get_device_properties(0).multi_processor_count // (B * H) + 1 if long else 2
    T = 128 * steps
    kc, ke, keep_k = _cache(ops, missing, twice, (T, B, H, 128), True, g)
    vc, ve, keep_v = _cache(ops, missing, twice, (T, B, H, 128), False, g)
    q = torch.randn(B, H * G, 128, device="cuda", generator=g).half()
    scaling = 0.25 / math.sqrt(128)
    for kw in (dict(), dict(splits=1, workspace=False)):
        out, st = ops.attn_decode(kc, vc, T, B, H, q, scaling, **kw)
        assert ops.read_status(st) == 0, kw
        s = torch.einsum("bhgd,tbhd->bhgt", q.double().view(B, H, G, 128), ke) * scaling
        want = torch.einsum("bhgt,tbhd->bhgd", torch.softmax(s, -1), ve).reshape(B, H * G, 128)
        # 1e-3 of the largest output, as for the attention everywhere (weights of 16 bits, fp16 outputs)
        assert float((out.double() - want).abs().max() / want.abs().max()) <= 1e-3, kw
