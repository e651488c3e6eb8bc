"""Operators called from several host threads."""
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
