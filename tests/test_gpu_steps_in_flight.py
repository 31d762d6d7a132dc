"""Decode steps one behind the other without a wait: the merge kernel runs beside the attention kernel, and the next step's attention kernel is set up beside both.
Each step finds the query and the newest row that the kernels ahead of it have written, and gives the bits that it gives when the host waits for everything in between."""
import pytest
import torch

from test_gpu_rounds import _cache, ops  # noqa: F401

pytestmark = pytest.mark.gpu


# launches of one round and of several, with one head and with groups; more heads than one launch takes; tails below and beyond a pass of 128 rows, and none
@pytest.mark.parametrize("T,B,Hkv,G,Tr", [(1024, 1, 32, 1, 100), (4096, 3, 32, 1, 130), (896, 2, 8, 4, 128), (2816, 3, 4, 6, 165), (4096, 8, 8, 4, 40),
                                          (640, 2, 3, 17, 129), (256, 1, 1, 2, 1), (16384, 1, 2, 8, 30), (1024, 2, 8, 2, 0),
                                          (5504, 2, 5, 3, 128), (3200, 2, 10, 4, 150)])         # (the merge kernel beside three or more workers)
def test_steps_without_a_wait(ops, T, B, Hkv, G, Tr):  # noqa: F811
    g = torch.Generator(device="cuda").manual_seed(T + G)
    kc, _, keep_k = _cache(ops, torch.randn(T, B, Hkv, 128, device="cuda", generator=g).half(), True, 0.05)
    vc, _, keep_v = _cache(ops, torch.randn(T, B, Hkv, 128, device="cuda", generator=g).half(), False, 0.1)
    steps = 12
    qs = torch.randn(steps, B, Hkv * G, 128, device="cuda", generator=g).half()
    ks, vs = (torch.randn(steps, B, Hkv, max(Tr, 1), 128, device="cuda", generator=g).half() for _ in range(2))
    one, zero = (torch.full((1, 1, 128), x, dtype=torch.float16, device="cuda") for x in (1.0, 0.0))
    ws, st = ops.attn_workspace(B, Hkv * G, ops.attn_splits(T, B, Hkv), "cuda"), ops.new_status("cuda")

    def run(wait):
        kt, vt = (torch.zeros(max(Tr, 1), B, Hkv, 128, dtype=torch.float16, device="cuda") for _ in range(2))
        q = torch.empty_like(qs[0])
        outs = []
        for i in range(steps):
            q.copy_(qs[i])
            if Tr:                                             # the last row by the kernel right ahead, the others by one before
                kt[:-1], vt[:-1] = ks[i, :, :, :-1].permute(2, 0, 1, 3), vs[i, :, :, :-1].permute(2, 0, 1, 3)
                ops.kv_store(ks[i, :, :, -1:].contiguous(), vs[i, :, :, -1:].contiguous(), one, zero, kt[-1:], vt[-1:])
            if wait:
                torch.cuda.synchronize()
            for _ in range(2):                                 # twice: a second layer's launch right behind the first's
                outs.append(ops.attn_decode(kc, vc, T, B, Hkv, q, 0.1, kt if Tr else None, vt if Tr else None, workspace=ws, status=st)[0])
                if wait:
                    torch.cuda.synchronize()
        return torch.stack(outs)
    want = run(True)
    for _ in range(3):
        assert torch.equal(run(False), want)
    assert ops.read_status(st) == 0
    assert torch.equal(want[0::2], want[1::2]) and not torch.equal(want[0], want[2])


@pytest.mark.parametrize("T,B,Hkv,G,Tr", [(1024, 1, 32, 1, 100), (5504, 2, 5, 3, 129), (0, 3, 4, 2, 300)])
def test_values_that_start_on_two_bytes(ops, T, B, Hkv, G, Tr):  # noqa: F811
    """The tail's values by 4-byte and by 2-byte loads, in launches with room beside the attention kernel's CTAs and without: the same bits."""
    g = torch.Generator(device="cuda").manual_seed(T + G)
    kc = vc = None
    if T:
        kc, _, keep_k = _cache(ops, torch.randn(T, B, Hkv, 128, device="cuda", generator=g).half(), True, 0.05)
        vc, _, keep_v = _cache(ops, torch.randn(T, B, Hkv, 128, device="cuda", generator=g).half(), False, 0.1)
    q = torch.randn(B, Hkv * G, 128, device="cuda", generator=g).half()
    kt, vt = (torch.randn(Tr, B, Hkv, 128, device="cuda", generator=g).half() for _ in range(2))
    odd = torch.empty(vt.numel() + 1, dtype=torch.float16, device="cuda")[1:].view(vt.shape)
    odd.copy_(vt)
    assert odd.data_ptr() % 4 == 2
    outs = [ops.attn_decode(kc, vc, T, B, Hkv, q, 0.1, kt, v)[0] for v in (vt, odd)]
    assert torch.equal(outs[0], outs[1]) and bool(torch.isfinite(outs[0]).all())


# one head and no tail: up to four workers in a CTA and more, in one round and in several
@pytest.mark.parametrize("T,B,Hkv", [(256, 1, 32), (4096, 2, 8), (4096, 1, 32), (8448, 4, 4), (4096, 3, 40)])
def test_steps_without_a_tail(ops, T, B, Hkv):  # noqa: F811
    test_steps_without_a_wait(ops, T, B, Hkv, 1, 0)
