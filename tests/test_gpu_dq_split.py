"""dQ pass of few, long items: a cluster shares the key tiles of a query tile (csrc/attn_bwd.cuh, dq_exchange)."""
import pytest
import torch

import modern_llm_v1_b200 as m

from gpu_util import check_against_oracle, randn_bf16, run_fwd_bwd
from test_gpu_parity import _case
from test_gpu_status_word import _full_cache, _nan_like, _overflow, _take_status, _untouched

pytestmark = pytest.mark.gpu

# CTAs per item 2, 2, 4, 4, 2 at D = 64 and 1, 2, 2, 4, 2 at D = 128; the first query tiles have fewer key tiles than the cluster CTAs
SHAPES = [(1, 1025, 8, 4), (1, 1900, 4, 2), (1, 2049, 2, 1), (1, 3011, 1, 1), (2, 2000, 2, 2)]


@pytest.mark.parametrize("B,T,Hq,Hkv", SHAPES)
@pytest.mark.parametrize("D", [64, 128])
def test_split_dq(B, T, Hq, Hkv, D):
    got, _ = check_against_oracle(*_case(B, T, Hq, Hkv, D), layout="BTHD" if T & 1 else "BHTD")
    again = run_fwd_bwd(*_case(B, T, Hq, Hkv, D), layout="BTHD" if T & 1 else "BHTD")
    assert all(torch.equal(a, b) for a, b in zip(got, again)), "a call does not repeat bit for bit"


@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 1900, 4, 2), (1, 3011, 1, 1)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("where", ["key", "query", "value", "gradient"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nan_and_infinity_go_where_an_unshared_item_takes_them(B, T, Hq, Hkv, D, where, bad):
    # the same sequence sixteen times: too many items to share any
    q, k, v, do = _case(B, T, Hq, Hkv, D)
    x = {"key": k, "query": q, "value": v, "gradient": do}[where]
    x[0, 0, T // 2, 5] = bad
    got = [y.float() for y in run_fwd_bwd(q, k, v, do)]
    want = [y[:1].float() for y in run_fwd_bwd(*(y.repeat(16, 1, 1, 1) for y in (q, k, v, do)))]
    for a, w in zip(got, want):
        assert torch.equal(torch.isfinite(a), torch.isfinite(w)) and torch.equal(torch.isnan(a), torch.isnan(w))
    assert not torch.isfinite(got[2][0, 0]).all()  # it reached dQ of its head
    assert Hkv == 1 or torch.isfinite(got[2][0, Hq // Hkv :]).all()


@pytest.mark.parametrize("D", [64, 128])
def test_a_set_status_word_leaves_dq_alone(D):
    B, T, Hq, Hkv = 1, 3000, 2, 1
    q, k, v, do = (randn_bf16((B, h, T, D), s) for s, h in ((1, Hq), (2, Hkv), (3, Hkv), (4, Hq)))
    o, lse = torch.empty_like(q), torch.empty((B, Hq, T), device="cuda")
    m.flash_attn_forward_gqa(q, k, v, o, lse, B, T, Hq, Hkv, D)
    c = _full_cache()
    m.device_status()
    dq, dk, dv = _nan_like(q, k, v)
    _overflow(c)
    m.flash_attn_backward_gqa(q, k, v, o, lse, do, dq, dk, dv, B, T, Hq, Hkv, D)
    _take_status()
    assert _untouched(dq, dk, dv)
    m.flash_attn_backward_gqa(q, k, v, o, lse, do, dq, dk, dv, B, T, Hq, Hkv, D)
    m.device_status()
    assert all(torch.isfinite(x.float()).all().item() for x in (dq, dk, dv))
