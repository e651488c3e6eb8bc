"""Scratch memory of the operators.  Operators called from several host threads, all on one CUDA stream (every thread's default): an operator's launches may not
have another call's between them while they share scratch memory.  A captured backward keeps its scratch when the stream's buffer grows."""
import threading

import pytest
import torch

import modern_llm_v1_b200 as m

from gpu_util import randn_bf16

pytestmark = pytest.mark.gpu


def test_an_operator_may_be_the_first_cuda_call_of_a_thread():
    B, T, Hq, Hkv, D = 1, 200, 2, 1, 64
    q, k, v = (randn_bf16((B, h, T, D), s) for s, h in ((1, Hq), (2, Hkv), (3, Hkv)))
    out = [(torch.empty_like(q), torch.empty((B, Hq, T), device="cuda")) for _ in range(2)]
    errors = []

    def run(i):
        try:
            m.flash_attn_forward_gqa(q, k, v, *out[i], B, T, Hq, Hkv, D)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    run(0)
    t = threading.Thread(target=run, args=(1,))
    t.start()
    t.join()
    m.device_status()
    assert not errors
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


def test_backward_beside_other_operators_of_other_threads():
    B, T, Hq, Hkv, D, n = 2, 300, 6, 2, 64, 300
    q, k, v, do = (randn_bf16((B, h, T, D), s) for s, h in ((1, Hq), (2, Hkv), (3, Hkv), (4, Hq)))
    o, lse = torch.empty_like(q), torch.empty((B, Hq, T), device="cuda")
    m.flash_attn_forward_gqa(q, k, v, o, lse, B, T, Hq, Hkv, D)
    outs = [[(torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)) for _ in range(n)] for _ in range(2)]

    # caches whose partial results fill the scratch, of sizes that make it grow while the others run
    caches = [(randn_bf16((1, 2, 64), 5), randn_bf16((1, 1, L, 64), 6), randn_bf16((1, 1, L, 64), 7)) for L in (9000, 30000, 70000)]
    x, g = randn_bf16((B, T, Hq, D), 8), torch.ones(D, device="cuda")
    cos, sin = m.make_rope_cache(T, D)
    y, rstd = torch.empty_like(q), torch.empty((B, Hq, T), device="cuda")
    m.rope_qknorm_forward(x, cos, sin, g, 1e-5, y, rstd, B, T, Hq, D)
    dx, dg = torch.empty_like(x), torch.zeros(D, device="cuda")
    m.device_status()
    errors = []

    def guarded(fn):
        def run():
            try:
                fn()
            except Exception as e:  # noqa: BLE001
                errors.append(e)
        return threading.Thread(target=run)

    def backward(i):
        for dq, dk, dv in outs[i]:
            m.flash_attn_backward_gqa(q, k, v, o, lse, do, dq, dk, dv, B, T, Hq, Hkv, D)

    def others():
        for i in range(n):
            cq, ck, cv = caches[i * 3 // n]
            m.flash_attn_decode(cq, ck, cv, torch.empty_like(cq), None, 1, ck.shape[2], 2, 1, 64)
            m.rope_qknorm_backward(do, x, cos, sin, g, rstd, dx, dg, B, T, Hq, D)

    threads = [guarded(lambda: backward(0)), guarded(others), guarded(lambda: backward(1))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    m.device_status()
    assert not errors
    want = tuple(torch.empty_like(t) for t in (q, k, v))
    m.flash_attn_backward_gqa(q, k, v, o, lse, do, *want, B, T, Hq, Hkv, D)
    m.device_status()
    wrong = sum(not torch.equal(a, b) for side in outs for got in side for a, b in zip(got, want))
    assert wrong == 0, f"{wrong} of {2 * 3 * n} gradients differ"


def test_a_captured_backward_keeps_its_scratch():
    B, T, Hq, Hkv, D = 1, 256, 2, 1, 64
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        q, k, v, do = (randn_bf16((B, h, T, D), s) for s, h in ((1, Hq), (2, Hkv), (3, Hkv), (4, Hq)))
        o, lse = torch.empty_like(q), torch.empty((B, Hq, T), device="cuda")
        m.flash_attn_forward_gqa(q, k, v, o, lse, B, T, Hq, Hkv, D)
        grads = tuple(torch.empty_like(t) for t in (q, k, v))
        run = lambda: m.flash_attn_backward_gqa(q, k, v, o, lse, do, *grads, B, T, Hq, Hkv, D)
        run()
        m.device_status()
        want = tuple(t.clone() for t in grads)
        graph = torch.cuda.CUDAGraph()
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            run()
        # larger problems on the same stream outgrow the buffer the graph writes its row vectors to; whatever is allocated
        # then may not lie in it
        for n in (2, 8, 64):
            big = [randn_bf16((n, h, T, D), s) for s, h in ((1, Hq), (2, Hkv), (3, Hkv), (4, Hq))]
            bo, bl = torch.empty_like(big[0]), torch.empty((n, Hq, T), device="cuda")
            m.flash_attn_forward_gqa(*big[:3], bo, bl, n, T, Hq, Hkv, D)
            m.flash_attn_backward_gqa(*big[:3], bo, bl, big[3], *(torch.empty_like(t) for t in big[:3]), n, T, Hq, Hkv, D)
            del big, bo, bl
            others = [torch.full((size,), 7, dtype=torch.uint8, device="cuda") for size in (4096, 8192, 16384, 65536) for _ in range(50)]
            for t in grads:
                t.fill_(float("nan"))
            graph.replay()
            side.synchronize()
            assert all((t == 7).all().item() for t in others)
            assert all(torch.equal(a, b) for a, b in zip(grads, want))
    m.device_status()
