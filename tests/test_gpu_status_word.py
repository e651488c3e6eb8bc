"""While the device status word is set, no attention kernel writes its outputs (include/b200attn.h).  The word is set here the
way a program would meet it, by an append beyond a cache's capacity (code 105): no kernel waits for anything that never comes."""
import pytest
import torch

import modern_llm_v1_b200 as m

from gpu_util import randn_bf16

pytestmark = pytest.mark.gpu


def _full_cache():
    """A cache whose device-side position says "full" behind the host's back; _overflow() then sets the status word."""
    cache = m.KVCache(1, 1, 1, 1, 64, 4)
    cache.set_lengths([3])
    cache.lengths[0] = 4
    x, g = torch.zeros((1, 1, 1, 64), device="cuda"), torch.ones(64, device="cuda")
    return cache, x, g, torch.empty((1, 1, 1, 64), dtype=torch.bfloat16, device="cuda")


def _overflow(c):
    cache, x, g, q = c
    cache.append(0, x, x, x, g, g, q)


def _take_status():
    with pytest.raises(RuntimeError, match="exceeds the cache capacity"):
        m.device_status()
    assert m.device_status() == 0


def _nan_like(*ts):
    return [torch.full_like(t, float("nan")) for t in ts]


def _untouched(*ts):
    return all(torch.isnan(t.float()).all().item() for t in ts)


# an item of its own per CTA and items shared by 2, 4 or 8 CTAs (forward, dK/dV pass), at both head dimensions
SHAPES = [(32, 512, 6, 2, 64), (1, 2000, 6, 2, 64), (1, 3000, 1, 1, 64), (1, 700, 8, 1, 64),
          (8, 1001, 16, 4, 128), (1, 2000, 4, 2, 128), (1, 3000, 1, 1, 128)]


@pytest.mark.parametrize("B,T,Hq,Hkv,D", SHAPES)
@pytest.mark.parametrize("mode", ["two_pass", "one_pass"])
def test_a_set_status_word_leaves_the_outputs_of_forward_and_backward_alone(B, T, Hq, Hkv, D, mode):
    if mode == "one_pass" and D != 64:
        pytest.skip("the one-pass backward is a D = 64 kernel")
    q, k, v, do = (randn_bf16((B, h, T, D), s) for s, h in ((1, Hq), (2, Hkv), (3, Hkv), (4, Hq)))
    o0, l0 = torch.empty_like(q), torch.empty((B, Hq, T), device="cuda")
    m.flash_attn_forward_gqa(q, k, v, o0, l0, B, T, Hq, Hkv, D)
    c = _full_cache()
    m.device_status()
    o, lse, dq, dk, dv = _nan_like(q, l0, q, k, v)
    _overflow(c)
    m.flash_attn_forward_gqa(q, k, v, o, lse, B, T, Hq, Hkv, D)
    m.flash_attn_backward_gqa(q, k, v, o0, l0, do, dq, dk, dv, B, T, Hq, Hkv, D, mode=mode)
    _take_status()
    assert _untouched(o, lse), "the forward wrote"
    assert _untouched(dq), "the dQ pass wrote"
    assert _untouched(dk, dv), "the dK/dV pass wrote"
    # and with the word cleared the same calls work
    m.flash_attn_forward_gqa(q, k, v, o, lse, B, T, Hq, Hkv, D)
    m.flash_attn_backward_gqa(q, k, v, o, lse, do, dq, dk, dv, B, T, Hq, Hkv, D, mode=mode)
    m.device_status()
    assert torch.equal(o, o0) and torch.equal(lse, l0)
    assert all(torch.isfinite(x.float()).all().item() for x in (dq, dk, dv))


@pytest.mark.parametrize("B,L,Hq,Hkv,D", [(1, 1025, 4, 2, 64), (1, 1500, 16, 4, 128), (120, 130, 6, 3, 64), (1, 30001, 2, 1, 64)])
def test_a_set_status_word_leaves_the_outputs_of_the_decode_alone(B, L, Hq, Hkv, D):
    q, kc, vc = randn_bf16((B, Hq, D), 1), randn_bf16((B, Hkv, L, D), 2), randn_bf16((B, Hkv, L, D), 3)
    c = _full_cache()
    m.device_status()
    o, lse = _nan_like(q, torch.empty((B, Hq), device="cuda"))
    _overflow(c)
    m.flash_attn_decode(q, kc, vc, o, lse, B, L, Hq, Hkv, D)
    _take_status()
    assert _untouched(o, lse)
    m.flash_attn_decode(q, kc, vc, o, lse, B, L, Hq, Hkv, D)
    m.device_status()
    assert torch.isfinite(o.float()).all() and torch.isfinite(lse).all()


@pytest.mark.parametrize("T,D", [(16384, 64), (16384, 128)])
def test_a_word_set_while_the_dq_pass_runs_keeps_the_dkdv_pass_from_writing(T, D):
    # The dK/dV pass's CTAs get in under the dQ pass (which leaves SMs free here and runs for hundreds of microseconds) and
    # read the word while it is clear.  Everything is enqueued behind one event, so the host's pace does not matter.
    B, Hq, Hkv = 1, 1, 1
    q, k, v, do = (randn_bf16((B, 1, T, D), s) for s in (1, 2, 3, 4))
    o, lse = torch.empty_like(q), torch.empty((B, Hq, T), device="cuda")
    m.flash_attn_forward_gqa(q, k, v, o, lse, B, T, Hq, Hkv, D)
    dq, dk, dv = _nan_like(q, k, v)
    # (of higher priority: its block must not queue behind the dK/dV pass's, which wait for SMs)
    main, other, gate = torch.cuda.current_stream(), torch.cuda.Stream(priority=-1), torch.cuda.Stream()
    c = _full_cache()
    # (a backward allocates its scratch on its first call)
    m.flash_attn_backward_gqa(q, k, v, o, lse, do, torch.empty_like(q), torch.empty_like(k), torch.empty_like(v), B, T, Hq, Hkv, D)
    m.device_status()
    go = torch.cuda.Event()
    with torch.cuda.stream(gate):
        torch.cuda._sleep(4_000_000)  # about 2 ms, for the host to enqueue what follows
        go.record()
    with torch.cuda.stream(other):
        other.wait_event(go)
        torch.cuda._sleep(60_000)  # about 30 us into the dQ pass
        _overflow(c)
    main.wait_event(go)
    m.flash_attn_backward_gqa(q, k, v, o, lse, do, dq, dk, dv, B, T, Hq, Hkv, D)
    main.wait_stream(other)
    main.synchronize()
    _take_status()
    assert _untouched(dk, dv)
