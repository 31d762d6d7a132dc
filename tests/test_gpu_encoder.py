"""Many blocks and alphabets around the sizes at which the encoder changes its way of looking symbols up."""
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


@pytest.mark.parametrize("is_k,nsym", [(True, 31), (False, 32), (True, 33), (False, 129)])
def test_encoder_with_many_blocks_and_symbols(ops, is_k, nsym):
    T, B, H = (1024, 8, 40) if is_k else (2048, 8, 20)    # 5120 blocks
    rng = np.random.default_rng(nsym)
    p = np.exp(-((np.arange(nsym) - nsym / 2) / (nsym / 5)) ** 2) + 1e-5
    part = rng.choice(nsym, size=(T // 8, B, H, 128), p=p / p.sum()).astype(np.uint8)
    part.reshape(-1)[:997 * nsym:997] = np.arange(nsym)    # every symbol, the rare ones not in one vector
    codes = np.concatenate([part] * 8)
    oenc, _ = orc.gen_codes(orc.histogram(codes))
    odata, obi, oti, _ = orc.encode(codes, is_k, oenc)
    dcodes = torch.from_numpy(codes).cuda()
    book = ops.build_codebook(ops.histogram(dcodes.view(-1)))
    bsz, tsz, _, cap = ops.buffer_sizes(T, B * H * 128, is_k)
    bi, ti = torch.zeros(bsz, dtype=torch.uint8, device="cuda"), torch.zeros(tsz // 2, dtype=torch.int16, device="cuda")
    enc = torch.zeros(cap, dtype=torch.uint8, device="cuda")
    total, st = ops.encode(dcodes, is_k, book.encode_table(), bi, ti, enc)
    assert ops.read_status(st) == 0 and int(total[0]) == odata.size
    assert np.array_equal(enc[:odata.size].cpu().numpy(), odata)
    assert np.array_equal(bi.cpu().numpy(), obi) and np.array_equal(ti.cpu().numpy().view(np.uint16), oti)
