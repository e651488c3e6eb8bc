"""The next kernel of a stream may start while a forward or backward works on its last items: calls that feed one another give what
they give with a synchronisation in between."""
import pytest
import torch

import modern_llm_v1_b200 as m

from gpu_util import randn_bf16

pytestmark = pytest.mark.gpu

# a CTA per SM at most; two; several items per CTA; clusters of every size; one tile per sequence by head and by group
SHAPES = [(8, 300, 6, 2), (14, 300, 6, 2), (36, 300, 6, 2), (2, 1000, 4, 2), (1, 2000, 4, 4), (1, 2500, 2, 1), (2, 128, 6, 2), (20, 128, 6, 2),
          (14, 100, 6, 2), (60, 128, 4, 4)]


@pytest.mark.parametrize("B,T,Hq,Hkv", SHAPES)
@pytest.mark.parametrize("D", [64, 128])
def test_calls_in_a_row(B, T, Hq, Hkv, D):
    def run(sync):  # each call reads what the one in front wrote
        q, k, v = (randn_bf16((B, h, T, D), s) for s, h in ((1, Hq), (2, Hkv), (3, Hkv)))
        n = 6
        bufs = [(torch.empty_like(q), torch.empty((B, Hq, T), device="cuda"), torch.empty_like(q), torch.empty_like(k), torch.empty_like(v))
                for _ in range(n)]
        do = randn_bf16((B, Hq, T, D), 4)
        torch.cuda.synchronize()
        for o, lse, dq, dk, dv in bufs:
            m.flash_attn_forward_gqa(q, k, v, o, lse, B, T, Hq, Hkv, D)
            if sync:
                torch.cuda.synchronize()
            m.flash_attn_backward_gqa(q, k, v, o, lse, do, dq, dk, dv, B, T, Hq, Hkv, D)
            if sync:
                torch.cuda.synchronize()
            q, k, v = dq, dk, dv
        return [x for b in bufs for x in b]

    want = run(True)
    for _ in range(3):
        for got, w in zip(run(False), want):
            assert torch.equal(got.view(torch.uint8), w.view(torch.uint8))
    m.device_status()
