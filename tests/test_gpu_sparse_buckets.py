"""Scalars that leave most buckets empty (0 and 1, one bit, all zero): whole warps of
the quad kernels then meet nothing but identities.  The bases repeat 300 points, so
that the oracle's MSM is over 300 summed scalars."""

import numpy as np
import pytest
import torch

import helioselene_gb300 as hs
import oracle
from conftest import oracle_inputs

pytestmark = pytest.mark.gpu

K = 300


@pytest.fixture(scope="module")
def bases():
    return {c: oracle_inputs(c, K, seed=41 + c)[1].reshape(K, 64) for c in (0, 1)}


def scalars(kind, n):
    rng = np.random.default_rng(n)
    s = np.zeros((n, 32), np.uint8)
    if kind == "bits":
        s[:, 0] = rng.integers(0, 2, n)
    elif kind == "one_power":  # one bit below 2^240: 70000 of them stay below 2^256
        b = rng.integers(0, 239, n)
        s[np.arange(n), b // 8] = 1 << (b % 8)
    elif kind == "one_bucket":
        s[:, 3] = 5
    return s


def expected(curve, s, idx, bases):
    sums = [0] * K
    for row, i in zip(s, idx):
        sums[i] += int.from_bytes(row.tobytes(), "little")
    sc = np.frombuffer(b"".join(v.to_bytes(32, "little") for v in sums), np.uint8)
    return oracle.msm(curve, sc.reshape(K, 32), bases, keep_carry=True)


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("kind", ["bits", "one_power", "one_bucket"])
# window sums by quads, by chunks and their sum; batches by chunks alone and by one quad a window
@pytest.mark.parametrize("n,count", [(3000, 1), (20000, 1), (70000, 1), (9000, 4), (150, 70)])
def test_sparse_buckets(ctx, bases, curve, kind, n, count):
    s = scalars(kind, n * count)
    rng = np.random.default_rng(count)
    idx = rng.integers(0, K, n * count)
    d_s = torch.from_numpy(s.reshape(-1)).cuda()
    d_p = torch.from_numpy(np.ascontiguousarray(bases[curve][idx]).reshape(-1)).cuda()
    d_o = torch.zeros(32 * count, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ctx.msm_batch_device(curve, [n] * count, d_s.data_ptr(), d_p.data_ptr(), d_o.data_ptr(), hs.FMT_COMPRESSED)
    torch.cuda.ExternalStream(ctx.stream).synchronize()
    got = d_o.cpu().numpy().reshape(count, 32)
    for j in sorted({0, 1, count // 2, count - 1} & set(range(count))):
        lo, hi = j * n, (j + 1) * n
        assert got[j].tobytes() == expected(curve, s[lo:hi], idx[lo:hi], bases[curve]), j
