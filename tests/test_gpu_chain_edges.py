"""Equal and opposite operands inside the reduction and the window combination,
at window widths around the sizes of their blocks: buckets that hold the same
or opposite points (the running sums then double or cancel), and window sums
that meet the running total as an equal or an opposite point.  Results are
compared bit for bit with the oracle."""

import numpy as np
import pytest

import oracle
from conftest import oracle_inputs

pytestmark = pytest.mark.gpu

ORDER = {0: 2**255 - 85737960593035654572250192257530476641, 1: 2**255 - 19}


def enc(v: int) -> bytes:
    return (v % 2**256).to_bytes(32, "little")


def neg(pt: np.ndarray, curve: int) -> np.ndarray:
    m = ORDER[1 - curve]
    out = pt.copy()
    out[32:] = np.frombuffer((m - int.from_bytes(pt[32:].tobytes(), "little")).to_bytes(32, "little"), np.uint8)
    return out


def check(ctx, curve, scalars, points, c):
    sc = np.frombuffer(b"".join(scalars), np.uint8)
    pts = np.concatenate(points)
    ctx.set_window(curve, 0, 1 << 40, c)
    try:
        got = ctx.msm(curve, sc, pts)
    finally:
        ctx.set_window(curve, 0, 1, 0)
    assert got == oracle.msm(curve, sc, pts, keep_carry=True)


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("c", [4, 5, 7, 8, 9, 10, 13, 17, 20])
def test_equal_and_opposite_buckets(ctx, curve, c):
    _, pts, _ = oracle_inputs(curve, 4, 11)
    p, q = pts[0], pts[1]
    half = 1 << (c - 1)
    lows = sorted({1, 2, 3, 4, 5, 8, 9, half - 1, half} & set(range(1, half + 1)))
    # the same point in neighbouring buckets (doubling), then its opposite (cancelling), in two windows
    for shift in (0, c):
        check(ctx, curve, [enc(d << shift) for d in lows], [p] * len(lows), c)
        check(ctx, curve, [enc(d << shift) for d in lows for _ in (0, 1)],
              [x for d in lows for x in ((p, neg(p, curve)) if d % 2 else (p, q))], c)
    # every bucket of a window the same point
    n = min(half, 300)
    check(ctx, curve, [enc(d) for d in range(1, n + 1)], [p] * n, c)
    # opposite points in buckets d + 1 and d: the running sum is the identity at d
    check(ctx, curve, [enc(2), enc(1), enc(1)], [p, neg(p, curve), q], c)


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("c", [4, 8, 13, 16])
def test_window_sum_equal_or_opposite_to_the_total(ctx, curve, c):
    _, pts, _ = oracle_inputs(curve, 4, 13)
    p, r = pts[0], pts[2]
    big = ctx.scalar_mul(curve, np.frombuffer(enc(1 << c), np.uint8), p, out_fmt=2)  # 2^c p, affine
    for other in (big, neg(big, curve)):
        # total 2^c p meets +-2^c p in window 0, in window 1, and with another term after it
        check(ctx, curve, [enc(1 << c), enc(1)], [p, other], c)
        check(ctx, curve, [enc(1 << (2 * c)), enc(1 << c)], [p, other], c)
        check(ctx, curve, [enc(1 << (2 * c)), enc(1 << c), enc(3)], [p, other, r], c)
        check(ctx, curve, [enc(1 << (3 * c)), enc(1 << (2 * c)), enc(1 << c)], [p, other, r], c)
