"""Several work items per CTA, of one to three key tiles each: every role of the persistent kernels then crosses an item
boundary at every other step (the next item's products start under the previous item's last tile, its output rows leave
under the next one's first)."""
import pytest

from gpu_util import check_against_oracle
from test_gpu_parity import _case

pytestmark = pytest.mark.gpu


# items of the dQ pass: 960 of one 64-key tile; 960 of two (the second a single key); 720 of two or three; counter-based lists with 1920.
# "auto" takes the first two shapes at D = 128 to the kernel for sequences of one tile.
@pytest.mark.parametrize("B,T,Hq,Hkv", [(80, 40, 12, 4), (160, 65, 6, 2), (60, 130, 6, 3), (160, 129, 6, 6)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mode", ["auto", "two_pass"])
def test_short_items_in_a_row(B, T, Hq, Hkv, D, mode):
    check_against_oracle(*_case(B, T, Hq, Hkv, D), layout="BTHD" if T == 65 else "BHTD", mode=mode)
