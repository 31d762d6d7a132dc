"""What kvc_store_packed refuses, before it launches anything (CPU)."""
import pytest
import torch

from kvcomp_b200 import _lib, ops

WORDS = ("x cos sin cos_stride B H x_tokens T D block codes min_int scale scratch scratch_bytes book enc_codes enc_T base_offset block_info thread_info "
         "encoded encoded_capacity rest rest_rows kept kept_rows report enc_table").split()
INTS = "mode batch_shared heads is_k build min_bytes".split()


def _refusal(**change):
    """The call's message for a prompt of 200 tokens, 3 heads, 128 compressed, all pointers at one (never touched) place."""
    place = 1 << 20
    a = dict.fromkeys(WORDS, place)
    a.update(cos_stride=0, B=1, H=3, x_tokens=200, T=128, D=128, block=64, scratch_bytes=1 << 20, enc_T=128, base_offset=0, encoded_capacity=1 << 20,
             rest_rows=72, kept_rows=128, enc_table=0, mode=_lib.MODE_CHANNEL, batch_shared=0, heads=1, is_k=1, build=1, min_bytes=2)
    a.update(change)
    blob = _lib.STORE_ARGS.pack(*(a[n] for n in WORDS), *(a[n] for n in INTS), 0.05, 0)
    lib = _lib.load()
    assert lib.kvc_store_packed(blob, None) != _lib.KVC_OK
    return lib.kvc_last_error().decode()


@pytest.mark.parametrize("offset", [1 << 32, (5 << 32) + 64, -1])
def test_offsets_beyond_32_bits(offset):
    assert "32 bits" in _refusal(base_offset=offset)


@pytest.mark.parametrize("change, words", [
    (dict(rest_rows=73), "73 rows behind"), (dict(rest_rows=-1), "row counts"), (dict(heads=0), "72 rows behind"), (dict(rest=0), "72 rows behind"),
    (dict(kept_rows=129), "row counts"), (dict(kept_rows=-64), "row counts"), (dict(kept_rows=32), "whole units"), (dict(kept=0), "whole units"),
    (dict(T=0, build=0, kept_rows=0), "rows behind"), (dict(T=0, rest_rows=0, kept_rows=0), "nothing to build"), (dict(enc_T=-64), "bad shape")])
def test_rows_that_the_call_cannot_write(change, words):
    assert words in _refusal(**change)


@pytest.mark.parametrize("offset", [1 << 32, -1])
def test_the_encoders_refuse_them_too(monkeypatch, offset):
    monkeypatch.setattr(ops, "_cuda", lambda t, dtype, name: t)
    codes = torch.zeros(64, 1, 1, 128, dtype=torch.uint8)
    buf = torch.zeros(8192, dtype=torch.uint8)
    for call in (ops.encode, ops.encode_now):
        with pytest.raises(_lib.KvcError, match="32 bits"):
            call(codes, True, buf, buf, buf, buf, base_offset=offset)


def test_a_call_for_nothing():
    """No token and no code: kvc_encode refused such a call, as a tensor without elements has no address."""
    assert "nothing to store" in _refusal(T=0, enc_T=0, build=0, rest_rows=0, kept_rows=0)
