"""The window combination by groups of windows: at every border between groups, a
total that equals or opposes the next group's sum, groups with nothing in them, and
groups whose own windows cancel, at widths that give eight, five and three groups."""

import numpy as np
import pytest

from conftest import oracle_inputs
from test_gpu_chain_edges import check, enc, neg

pytestmark = pytest.mark.gpu

GROUPS = {8: 8, 10: 5, 16: 5, 20: 3}


def borders(c):
    w = (257 + c - 1) // c
    per = -(-w // GROUPS[c])
    return [w - j * per for j in range(1, GROUPS[c]) if w - j * per > 0]


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("c", sorted(GROUPS))
def test_equal_or_opposite_at_each_border(ctx, curve, c):
    _, pts, _ = oracle_inputs(curve, 4, 29)
    p, r = pts[0], pts[2]
    for b in borders(c):
        # the groups from window b up sum to p (a digit of 1 in window b), which meets
        # +-2^(c k) p, a digit of 1 in window b - k, as the next group's whole sum
        for k in (1, min(2, b)):
            if c * k > 250:
                continue
            big = ctx.scalar_mul(curve, np.frombuffer(enc(1 << (c * k)), np.uint8), p, out_fmt=2)
            for other in (big, neg(big, curve)):
                check(ctx, curve, [enc(1 << (c * b)), enc(1 << (c * (b - k)))], [p, other], c)
                check(ctx, curve, [enc(1 << (c * b)), enc(1 << (c * (b - k))), enc(1)], [p, other, r], c)


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("c", sorted(GROUPS))
def test_empty_and_cancelling_groups(ctx, curve, c):
    _, pts, _ = oracle_inputs(curve, 4, 31)
    p, r = pts[0], pts[2]
    big = ctx.scalar_mul(curve, np.frombuffer(enc(1 << c), np.uint8), p, out_fmt=2)
    for b in borders(c):
        # only one group holds anything, then only its lowest window and window 0
        check(ctx, curve, [enc(1 << (c * b))], [p], c)
        check(ctx, curve, [enc(1 << (c * b)), enc(5)], [p, r], c)
        # two windows of one group cancel, alone and with terms above and below
        check(ctx, curve, [enc(1 << (c * (b + 1) if c * (b + 1) < 255 else c * b)), enc(1 << (c * b))],
              [p, neg(big, curve)], c)
        check(ctx, curve, [enc(1 << (c * b)), enc(1 << (c * (b - 1))), enc(3)], [p, neg(big, curve), r], c)
        if b >= 2:
            lo = [enc(1 << (c * (b - 1))), enc(1 << (c * (b - 2))), enc(7)]
            check(ctx, curve, lo, [p, neg(big, curve), r], c)
            check(ctx, curve, [enc(1 << (c * b))] + lo, [r, p, neg(big, curve), r], c)
