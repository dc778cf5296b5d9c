"""The second level of the reduction by one quad per window: thousands of windows of
one, two and more groups, mixed widths in one plan, empty MSMs, and buckets that all
hold the same point (the running sums then double)."""

import numpy as np
import pytest
import torch

import helioselene_gb300 as hs
import oracle
from conftest import oracle_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("window", [4, 6, 8, 10])  # 2047 windows: the block per window; from 2048 the quad
def test_commitments(ctx, curve, window):
    n, count = 3, 2053
    _, G, _ = oracle_inputs(curve, n, seed=7)
    rng = np.random.default_rng(window)
    vals = rng.integers(0, 256, (count, n, 32), dtype=np.uint8)
    vals[0], vals[1] = 255, 0
    vals[2] = 0
    vals[2, :, 0] = [1, 2, 3]
    fb = hs.FixedBase(ctx, curve, G, window=window)
    try:
        got = fb.commit(vals)
        assert got[:2047] == fb.commit(vals[:2047])
        for j in (0, 1, 2, 3, 1000, count - 1):
            assert got[j] == oracle.msm(curve, vals[j], G, keep_carry=True), j
    finally:
        fb.close()


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("kind", ["random", "same_point", "edges"])
def test_mixed_batch(ctx, curve, kind):
    top = 2000
    sc, pts, _ = oracle_inputs(curve, top, seed=53 + curve)
    sc, pts = sc.reshape(top, 32).copy(), pts.reshape(top, 64).copy()
    if kind == "same_point":
        pts[:] = pts[0]
    elif kind == "edges":
        sc[::3] = 0
        sc[1::3] = 255
    edges = [0, 1, 30, 161, 501, 1601, top]
    sizes = [edges[i % len(edges)] for i in range(100)]
    d_s = torch.from_numpy(np.concatenate([sc[:n] for n in sizes]).reshape(-1)).cuda()
    d_p = torch.from_numpy(np.concatenate([pts[:n] for n in sizes]).reshape(-1)).cuda()
    d_o = torch.zeros(32 * len(sizes), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    ctx.msm_batch_device(curve, sizes, d_s.data_ptr(), d_p.data_ptr(), d_o.data_ptr(), hs.FMT_COMPRESSED)
    torch.cuda.ExternalStream(ctx.stream).synchronize()
    got = d_o.cpu().numpy().reshape(-1, 32)
    want = {n: oracle.msm(curve, sc[:n], pts[:n], keep_carry=True) for n in edges if n}
    want[0] = ctx.msm(curve, np.zeros((1, 32), np.uint8), pts[:1])
    for i, n in enumerate(sizes):
        assert got[i].tobytes() == want[n], (i, n)
