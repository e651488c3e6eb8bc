"""The comparison that the strong-scaling block of bench.py makes between the ranks' gathered outputs and the whole run."""
import pytest
import torch

from modern_llm_v1_b200 import sharding


def _gradient(seed, std):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn((6, 3, 300, 64), generator=g) * std).bfloat16()  # T: two tiles of 128 and a rest


@pytest.mark.parametrize("std", [1.0, 1e-3])
def test_one_step_of_rounding_passes_and_a_wrong_row_does_not(std):
    want = _gradient(1, std)
    # a third of the elements one BF16 step off
    bits = want.view(torch.int16).clone()
    bits[..., ::3] += 1
    flipped = bits.view(torch.bfloat16)
    assert 0 < sharding.worst_tile_rel_l2(flipped, want) <= sharding.TILE_REL_L2
    assert sharding.worst_tile_rel_l2(want, want) == 0
    # one row of one tile, at the tiles' edges and in the rest
    for t in (0, 127, 128, 299):
        wrong = want.clone()
        wrong[4, 1, t] = 0
        assert sharding.worst_tile_rel_l2(wrong, want) > 10 * sharding.TILE_REL_L2


def test_a_nan_or_a_missing_tile_never_passes():
    want = _gradient(2, 1.0)
    for value in (float("nan"), float("inf")):
        bad = want.clone()
        bad[5, 2, 299, 63] = value
        assert not sharding.worst_tile_rel_l2(bad, want) <= sharding.TILE_REL_L2
    zero = want.clone()
    zero[0, 0, 128:256] = 0
    assert not sharding.worst_tile_rel_l2(want, zero) <= sharding.TILE_REL_L2
    assert sharding.worst_tile_rel_l2(zero, zero) == 0
