"""Small plans: the single-block sort against the general one (the same MSM in a
batch of two) and against the oracle, at point counts around a block's threads and
a segment's length and widths around the limits of the small plan; buckets that
hold every point; host buffers, whose bases arrive beside the sort."""

import numpy as np
import pytest

import helioselene_gb300 as hs
import oracle
from conftest import oracle_inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def own_ctx():
    c = hs.Context(0)
    yield c
    c.close()


def inputs(curve, n, kind):
    sc, pts, _ = oracle_inputs(curve, n, seed=17 * n + curve)
    sc = sc.copy()
    if kind == "one_bucket":  # every scalar the same: a bucket of n entries in every window
        sc[:] = sc[0]
    elif kind == "edges":
        sc[::3] = 0
        sc[1::3] = 255  # 2^256 - 1: the carry reaches the top window
    return sc, pts


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("kind", ["random", "one_bucket", "edges"])
@pytest.mark.parametrize("n", [1, 2, 8, 9, 16, 63, 65, 600, 1023, 1025, 2978, 2979])
def test_single_against_batch_and_oracle(own_ctx, curve, kind, n):
    sc, pts = inputs(curve, n, kind)
    want = oracle.msm(curve, sc, pts, keep_carry=True)
    own_ctx.set_window(curve, 0, 1, 0)
    assert own_ctx.msm(curve, sc, pts) == want  # from host buffers
    both = own_ctx.msm_batch([(curve, sc, pts), (curve, sc[:1], pts[:1])])
    assert both[0] == want


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("c,n", [(4, 1), (4, 100), (4, 1500), (5, 33), (6, 2000), (7, 64), (9, 16), (9, 3300), (10, 20)])
def test_widths(own_ctx, curve, c, n):
    own_ctx.set_window(curve, 0, 1 << 40, c)
    try:
        for kind in ("random", "one_bucket", "edges"):
            sc, pts = inputs(curve, n, kind)
            assert own_ctx.msm(curve, sc, pts) == oracle.msm(curve, sc, pts, keep_carry=True), kind
    finally:
        own_ctx.set_window(curve, 0, 1, 0)


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("n,c", [(1, 4), (18, 8), (38, 12), (228, 13), (500, 14)])
def test_one_fixed_base_commitment(own_ctx, curve, n, c):
    sc, pts = inputs(curve, n, "random")
    fb = hs.FixedBase(own_ctx, curve, pts, window=c)
    try:
        assert fb.commit(sc.reshape(-1))[0] == oracle.msm(curve, sc, pts, keep_carry=True)
    finally:
        fb.close()


def test_repeated_host_calls_of_changing_inputs(own_ctx):
    """the bases of a call are read only once they have arrived (the sort alone is
    shorter than their way to the device)"""
    for curve in (0, 1):
        for n in (700, 2900):
            data = [inputs(curve, n, "random") for _ in range(1)] + [
                (inputs(curve, n + 1, "random")[0][1:], inputs(curve, n + 1, "random")[1][1:])]
            want = [oracle.msm(curve, s, p, keep_carry=True) for s, p in data]
            for _ in range(20):
                for (s, p), w in zip(data, want):
                    assert own_ctx.msm(curve, s, p) == w
