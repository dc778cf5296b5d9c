"""The block sort of batches of small fixed-base MSMs (a block per commitment, its
buckets and list in shared memory) against the oracle: generator counts around a
block's threads and the entries it holds, few and many buckets, padded lists, scalars
that fill one bucket, are zero or have every bit set."""

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


# 128 commitments are the least; 20480 entries the most: 620 generators at 33 windows,
# 1024 at 20; 14 bits have too many buckets
@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("rounds", [-1, 0, 1, 2, 3])
@pytest.mark.parametrize("n,window,count", [(1, 0, 130), (17, 0, 130), (65, 8, 128), (65, 8, 127), (228, 0, 129),
                                            (620, 8, 128), (621, 8, 128), (1024, 13, 128), (1025, 13, 128),
                                            (130, 4, 128), (40, 14, 128)])
def test_commitments(own_ctx, curve, rounds, n, window, count):
    _, G, _ = oracle_inputs(curve, n, seed=n)
    rng = np.random.default_rng(n)
    vals = rng.integers(0, 256, (count, n, 32), dtype=np.uint8)
    vals[0] = 255
    vals[1] = 0
    vals[2:4] = vals[2, 0]
    fb = hs.FixedBase(own_ctx, curve, G, window=window)
    try:
        if rounds < 0:
            own_ctx.default_batch_affine()
        else:
            own_ctx.set_batch_affine(rounds, 0, curve)
        got = fb.commit(vals)
        for j in (0, 1, 2, 64, count - 1):
            assert got[j] == oracle.msm(curve, vals[j], G, keep_carry=True), j
        assert got[3] == got[2]
    finally:
        own_ctx.default_batch_affine()
        fb.close()


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("n,window,count", [(17, 0, 300), (228, 0, 256), (620, 8, 200)])
def test_every_commitment(own_ctx, curve, n, window, count):
    """all results of the block sort against those of calls of fewer commitments, which
    sort otherwise"""
    _, G, _ = oracle_inputs(curve, n, seed=3 * n)
    rng = np.random.default_rng(3 * n)
    vals = rng.integers(0, 256, (count, n, 32), dtype=np.uint8)
    vals[::9] = vals[::9, :1]
    vals[4::9, ::2] = 0
    fb = hs.FixedBase(own_ctx, curve, G, window=window)
    try:
        got = fb.commit(vals)
        for lo in range(0, count, 100):
            assert got[lo:lo + 100] == fb.commit(vals[lo:lo + 100]), lo
    finally:
        fb.close()
