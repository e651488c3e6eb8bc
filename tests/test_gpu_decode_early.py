"""A decode of many CTAs brings its first tiles into L2 while the kernel in front of it still runs.  What that kernel writes -
the newest row of the cache, the lengths - has to be what the decode computes with.  (Lengths that change under the look itself:
test_decode_walk_cpu.py.)"""
import pytest
import torch

import modern_llm_v1_b200 as m

from gpu_util import randn_bf16

pytestmark = pytest.mark.gpu


def _ragged(q, kc, vc, lens, ws):
    B, Hq, D = q.shape
    Hkv, L = kc.shape[1], kc.shape[2]
    o, lse = torch.full_like(q, float("nan")), torch.full((B, Hq), float("nan"), device="cuda")
    lib = m._lib.load()
    m._lib.check(lib.b200attn_decode_ragged(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), o.data_ptr(), lse.data_ptr(), lens.data_ptr(), B, L,
                                            L, Hq, Hkv, D, 0.0, 0, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), "decode")
    return o, lse


# 24 and 640 units: shares of a cluster on few CTAs, ranges and whole units on many; lengths of one tile up to the capacity.  The copies in
# front let the decode start only when they are complete, so its look finds the lengths and rows that they have just written.
@pytest.mark.parametrize("B,L,Hq,Hkv,D", [(6, 700, 8, 4, 64), (40, 1500, 8, 4, 64), (160, 300, 4, 4, 128), (40, 1500, 16, 4, 128)])
def test_what_the_kernel_in_front_writes_is_used(B, L, Hq, Hkv, D):
    q, kc, vc = randn_bf16((B, Hq, D), 61), randn_bf16((B, Hkv, L, D), 62), randn_bf16((B, Hkv, L, D), 63)
    true = torch.tensor([1 + (L - 1) * b // (B - 1) for b in range(B)], dtype=torch.int32, device="cuda")
    junk = torch.tensor([(-7, 0, 1 << 30, L, -(1 << 31), 3)[b % 6] for b in range(B)], dtype=torch.int32, device="cuda")
    lib = m._lib.load()
    ws = torch.empty(lib.b200attn_decode_workspace_bytes(B, L, Hq, Hkv, D, 0), dtype=torch.uint8, device="cuda")
    want_o, want_lse = _ragged(q, kc, vc, true, ws)
    torch.cuda.synchronize()
    lens, k2 = junk.clone(), torch.zeros_like(kc)
    for _ in range(5):
        lens.copy_(junk)
        k2.zero_()
        torch.cuda.synchronize()
        k2.copy_(kc)
        lens.copy_(true)
        o, lse = _ragged(q, k2, vc, lens, ws)
        assert torch.equal(o, want_o) and torch.equal(lse, want_lse)
    m.device_status()


# The append of one token lets the decode start while it writes: the look brings in first tiles (of two at most here) whose newest row is
# still to be written.  What stood there before would make every output NaN.
@pytest.mark.parametrize("B,L,Hq,Hkv,D", [(160, 200, 8, 4, 64), (300, 150, 4, 4, 64), (160, 120, 8, 2, 128), (64, 250, 4, 4, 128)])
@pytest.mark.parametrize("ragged", [False, True])
def test_the_row_that_the_append_in_front_writes_is_used(B, L, Hq, Hkv, D, ragged):
    lens = [1 + (L - 1) * b // (B - 1) if ragged else L for b in range(B)]
    kc, vc = randn_bf16((B, Hkv, L, D), 71), randn_bf16((B, Hkv, L, D), 72)
    for b, n in enumerate(lens):
        kc[b, :, n - 1] = vc[b, :, n - 1] = float("nan")
    xq, xk, xv = (randn_bf16((B, 1, h, D), s) for s, h in ((73, Hq), (74, Hkv), (75, Hkv)))
    gamma = torch.ones(D, device="cuda")
    cache = m.KVCache(1, B, Hq, Hkv, D, L)
    if ragged:
        cache.set_lengths([n - 1 for n in lens])
    else:
        cache.length = L - 1

    def step(sync):
        cache.k[0].copy_(kc)
        cache.v[0].copy_(vc)
        q = torch.full((B, Hq, 1, D), float("nan"), dtype=torch.bfloat16, device="cuda")
        o, lse = torch.full_like(q, float("nan")), torch.full((B, Hq, 1), float("nan"), device="cuda")
        torch.cuda.synchronize()
        cache.append(0, xq, xk, xv, gamma, gamma, q)
        if sync:
            torch.cuda.synchronize()
        cache.attend(0, q, o, lse)
        return o, lse

    want = step(True)
    assert all(torch.isfinite(x.float()).all() for x in want)
    for _ in range(10):
        assert all(torch.equal(a, b) for a, b in zip(step(False), want))
    m.device_status()
