"""Backward of sequences of at most one tile (csrc/attn_bwd_tile.cuh): a CTA per query head with the group as a cluster, or a CTA per
key/value head, against the oracle and the two passes."""
import pytest
import torch

import modern_llm_v1_b200 as m

from gpu_util import check_against_oracle, kernels_of, randn_bf16, run_fwd_bwd
from test_gpu_parity import _case
from test_gpu_status_word import _full_cache, _nan_like, _overflow, _take_status, _untouched

pytestmark = pytest.mark.gpu

# clusters of 1, 2, 3, 5, 6 and 8 query heads; by group at both D or at D = 128 only (several rounds of CTAs, a group larger than a
# cluster), where Q and dO of five heads and more go through two places; too few CTAs by group
GROUPS = {(3, 4, 4): "head head", (2, 4, 2): "head head", (2, 6, 2): "head head", (1, 5, 1): "head head", (2, 6, 1): "head head",
          (1, 16, 2): "head head", (60, 6, 2): "group group", (130, 8, 1): "group group", (50, 16, 4): "passes group",
          (180, 12, 1): "passes group", (24, 12, 1): "passes passes"}


@pytest.mark.parametrize("T", [1, 2, 33, 64, 127, 128])
@pytest.mark.parametrize("D", [64, 128])
def test_lengths_up_to_a_tile(T, D):
    check_against_oracle(*_case(2, T, 6, 2, D), layout="BTHD" if T & 1 else "BHTD")


@pytest.mark.parametrize("B,Hq,Hkv", GROUPS)
@pytest.mark.parametrize("D", [64, 128])
def test_groups_and_numbers_of_ctas(B, Hq, Hkv, D):
    got, _ = check_against_oracle(*_case(B, 100, Hq, Hkv, D))
    again = run_fwd_bwd(*_case(B, 100, Hq, Hkv, D))
    assert all(torch.equal(a, b) for a, b in zip(got, again)), "a call does not repeat bit for bit"
    # the same products in another grouping: a few roundings to BF16 (2^-9 each) of the outputs
    for a, b in zip(got[2:], run_fwd_bwd(*_case(B, 100, Hq, Hkv, D), mode="two_pass")[2:]):
        assert (a.float() - b.float()).norm() <= 2.0 ** -9 * b.float().norm()


@pytest.mark.parametrize("B,Hq,Hkv", GROUPS)
@pytest.mark.parametrize("D", [64, 128])
def test_which_kernel(B, Hq, Hkv, D):
    names = " ".join(n for n in kernels_of(lambda: run_fwd_bwd(*_case(B, 100, Hq, Hkv, D))) if "attn_bwd" in n)
    took = "head" if f"attn_bwd_tile_kernel<{D}, true>" in names else "group" if f"attn_bwd_tile_kernel<{D}, false>" in names else "passes"
    assert took == GROUPS[B, Hq, Hkv].split()[D == 128], names
    assert ("attn_bwd_dq" in names and "attn_bwd_dkdv" in names) == (took == "passes"), names


@pytest.mark.parametrize("B,Hq,Hkv", [(3, 4, 4), (60, 6, 2), (50, 16, 4)])
@pytest.mark.parametrize("D", [64, 128])
def test_heads_where_the_projection_left_them(B, Hq, Hkv, D):
    check_against_oracle(*_case(B, 77, Hq, Hkv, D), layout="BTHD")


# by head in a cluster, by head without a group, by group
@pytest.mark.parametrize("B,Hq,Hkv", [(2, 6, 2), (3, 4, 4), (60, 6, 2)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [100, 128])
@pytest.mark.parametrize("where", ["key", "query", "value", "gradient"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nan_and_infinity_go_where_the_two_passes_take_them(B, Hq, Hkv, D, T, where, bad):
    q, k, v, do = _case(B, T, Hq, Hkv, D)
    b, hk, group, row = B - 1, Hkv - 1, Hq // Hkv, 70
    x, h = {"key": (k, hk), "query": (q, hk * group), "value": (v, hk), "gradient": (do, hk * group)}[where]
    x[b, h, row, 5] = bad
    got = [y.float() for y in run_fwd_bwd(q, k, v, do)]
    want = [y.float() for y in run_fwd_bwd(q, k, v, do, mode="two_pass")]
    for a, w in zip(got, want):
        assert torch.equal(torch.isfinite(a), torch.isfinite(w)) and torch.equal(torch.isnan(a), torch.isnan(w))
    assert not torch.isfinite(got[3 if where == "value" else 4][b, hk]).all()  # it reached dK or dV of its head
    for i, own in enumerate((slice(hk * group, None),) * 3 + (slice(hk, None),) * 2):
        rest = got[i].clone()
        rest[b, own] = 0.0
        assert torch.isfinite(rest).all()


@pytest.mark.parametrize("B,Hq,Hkv", [(2, 6, 2), (3, 4, 4), (60, 6, 2)])
@pytest.mark.parametrize("D", [64, 128])
def test_a_set_status_word_leaves_the_gradients_alone(B, Hq, Hkv, D):
    T = 120
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
