"""How the fused dispatch + GEMM kernel's CTAs are dealt out (host arithmetic of the launcher)."""

import pytest

from lplb_b200 import _native

# (CTAs asked for, sender CTAs, pairs that fit at once) -> (tile CTAs, sender CTAs)
CASES = [
    ((148, 0, 74), (148, 0)), ((148, 16, 74), (132, 16)), ((148, 15, 74), (132, 16)), ((148, 147, 74), (2, 146)),
    ((147, 0, 74), (146, 0)), ((147, 1, 74), (144, 2)),  # an odd SM has no partner
    ((148, 0, 72), (144, 0)), ((148, 16, 70), (124, 16)), ((148, 147, 66), (2, 130)),  # fewer pairs fit than SMs / 2
    ((148, 16, 1), (2, 0)), ((2, 1, 74), (2, 0)),  # one pair: it runs tiles and its spare warps send
]


@pytest.mark.parametrize("asked,want", CASES)
def test_every_cta_of_the_launch_fits_at_once(asked, want):
    n_cta, send, resident = asked
    got = _native.load().moe_fused_grid(n_cta, send, resident)
    assert got == want
    assert sum(got) <= min(n_cta, 2 * resident) and got[0] >= 2
