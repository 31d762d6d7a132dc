"""The encoder of small alphabets: how many codes make one piece follows from the longest code (8, 13 bits), words are stored and only those that two vectors
share are ORed, and V's tile comes by 16 or by 4 bytes."""
import numpy as np
import pytest
import torch

from oracle import kvc_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("is_k", [True, False])
@pytest.mark.parametrize("longest", [1, 2, 7, 8, 9, 12, 13, 14, 16, 17])
@pytest.mark.parametrize("off", [0, 4])                      # the codes start on 16 bytes, or on 4
def test_longest_codes(is_k, longest, off):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops
    T, B, H = 256, 2, 3
    n = T * B * H * 128
    rng = np.random.default_rng(longest)
    nsym = longest + 1 if longest > 1 else 2                  # counts 2^i: a code of every length up to the longest, twice
    p = 2.0 ** -np.minimum(np.arange(1, nsym + 1), nsym - 1)
    codes = rng.choice(nsym, size=n, p=p).astype(np.uint8)
    codes[:nsym] = np.arange(nsym)
    v = codes.reshape(T, B, H, 128)
    v[:, 0, 0] = 0                                            # vectors of one bit a symbol, and of the longest codes alone
    long = rng.integers(max(0, nsym - 9), nsym, 128)
    v[130, 1, 2], v[128:, 0, 1, 5] = long, long               # (one of K's vectors, one of V's)
    counts = np.zeros(256, np.int64)
    counts[:nsym] = np.round(2.0 ** 40 * p)
    oenc, _ = orc.gen_codes(counts)
    assert int(oenc["length"].max()) == longest
    odata, obi, oti, _ = orc.encode(v, is_k, oenc)
    blob = torch.zeros(n + 16, dtype=torch.uint8, device="cuda")
    dcodes = blob[off:off + n].view(T, B, H, 128)
    dcodes.copy_(torch.from_numpy(v))
    table = torch.from_numpy(np.stack([oenc["code"], oenc["length"]], 1).astype("<u4").copy().view(np.uint8).reshape(-1)).cuda()
    bsz, tsz, _, cap = ops.buffer_sizes(T, B * H * 128, is_k)
    bi, ti = torch.zeros(bsz, dtype=torch.uint8, device="cuda"), torch.zeros(tsz // 2, dtype=torch.int16, device="cuda")
    for fill in (0, 255):                                     # whatever the stream's memory held
        enc = torch.full((2 * cap,), fill, dtype=torch.uint8, device="cuda")
        total, st = ops.encode(dcodes, is_k, table, bi, ti, enc)
        assert not ops.read_status(st, raise_on_fatal=False) & ~ops._lib.FLAG_VECTOR_LONG and int(total[0]) == odata.size
        assert np.array_equal(enc[:odata.size].cpu().numpy(), odata)
        assert np.array_equal(bi.cpu().numpy(), obi) and np.array_equal(ti.cpu().numpy().view(np.uint16), oti)


@pytest.mark.parametrize("is_k", [True, False])
@pytest.mark.parametrize("length", [32, 33, 36, 64, 1 << 31])
def test_codes_beyond_the_table(is_k, length):
    """A table entry has 32 bits for a code: a symbol whose code is longer has none, and is reported where it occurs."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from kvcomp_b200 import ops
    T, B, H = 128, 1, 2
    entries = np.zeros((256, 2), "<u4")
    entries[:3] = [[0, 1], [2, 2], [0xc0000000, length]]
    table = torch.from_numpy(entries.view(np.uint8).reshape(-1).copy()).cuda()
    bsz, tsz, _, cap = ops.buffer_sizes(T, B * H * 128, is_k)
    for used in (False, True):
        codes = torch.zeros(T, B, H, 128, dtype=torch.uint8, device="cuda")
        codes[5, 0, 1, 7] = 1
        if used:
            codes[T - 1, 0, H - 1, 127] = 2                   # the last vector's last symbol
        bi, ti, enc = (torch.zeros(n, dtype=torch.uint8, device="cuda") for n in (bsz, tsz, cap))
        total, st = ops.encode(codes, is_k, table, bi, ti, enc)
        flags = ops.read_status(st, raise_on_fatal=False)
        assert bool(flags & ops._lib.FLAG_SYMBOL_MISSING) == (used and length > 32)
        # a bit a symbol, two for the one, and 31 more for a code of 32 bits
        n = T * B * H * 16 + 1 + (4 if used and length == 32 else 0)
        assert int(total[0]) == n
