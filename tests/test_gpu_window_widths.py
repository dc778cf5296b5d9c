"""The default window widths: sizes on both sides of each border, alone, from host
encodings and in batches of few and many MSMs, against the same MSM at a width set
by hand, and against the oracle where the sizes are small."""

import numpy as np
import pytest
import torch

import helioselene_gb300 as hs
import oracle
from conftest import oracle_inputs

pytestmark = pytest.mark.gpu

_N = 350001


@pytest.fixture(scope="module")
def own_ctx():
    c = hs.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def large():
    """350001 bases per curve, 5000 of the oracle's repeated in a shuffled order, and scalars"""
    out = {}
    for curve in (0, 1):
        sc, pts, _ = oracle_inputs(curve, 5000, seed=70 + curve)
        rng = np.random.default_rng(curve)
        idx = rng.integers(0, 5000, _N)
        s = rng.integers(0, 256, (_N, 32), dtype=np.uint8)
        s[:, 31] &= 0x7F
        out[curve] = (s, np.ascontiguousarray(pts.reshape(5000, 64)[idx]))
    return out


def run_device(ctx, curve, s, p, sizes=None):
    d_s, d_p = torch.from_numpy(s.reshape(-1)).cuda(), torch.from_numpy(p.reshape(-1)).cuda()
    d_o = torch.zeros(32 * (len(sizes) if sizes else 1), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    if sizes:
        ctx.msm_batch_device(curve, sizes, d_s.data_ptr(), d_p.data_ptr(), d_o.data_ptr(), hs.FMT_COMPRESSED)
    else:
        ctx.msm_device(curve, d_s.data_ptr(), d_p.data_ptr(), s.shape[0], d_o.data_ptr(), hs.FMT_COMPRESSED)
    torch.cuda.ExternalStream(ctx.stream).synchronize()
    return d_o.cpu().numpy().reshape(-1, 32)


def at_width(ctx, curve, c, f):
    ctx.set_window(curve, 0, 1 << 40, c)
    try:
        return f()
    finally:
        ctx.set_window(curve, 0, 1, 0)


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("n", [10000, 10001, 24001, 48000, 48001, 80001, 350000, 350001])
def test_alone(own_ctx, large, curve, n):
    s, p = large[curve][0][:n], large[curve][1][:n]
    want = at_width(own_ctx, curve, 12, lambda: run_device(own_ctx, curve, s, p))
    assert (run_device(own_ctx, curve, s, p) == want).all()


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("n", [24001, 40001, 90001, 150001])
def test_host_encodings(own_ctx, large, curve, n):
    s, p = large[curve][0][:n], large[curve][1][:n]
    enc = own_ctx.compress(curve, p, hs.FMT_AFFINE)
    want = at_width(own_ctx, curve, 11, lambda: run_device(own_ctx, curve, s, p))
    assert own_ctx.msm(curve, s, enc, hs.FMT_COMPRESSED) == want.tobytes()


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("count", [63, 64])
def test_batches_of_few_and_many(own_ctx, curve, count):
    edges = [0, 1, 2, 159, 160, 161, 500, 501, 1600, 1601, 5000]
    sizes = [edges[i % len(edges)] for i in range(count)]
    sc, pts, _ = oracle_inputs(curve, 5000, seed=90 + curve, edge_fraction=0.05)
    sc, pts = sc.reshape(5000, 32), pts.reshape(5000, 64)
    s = np.concatenate([sc[:n] for n in sizes])
    p = np.concatenate([pts[:n] for n in sizes])
    got = run_device(own_ctx, curve, s, p, sizes)
    want = {n: oracle.msm(curve, sc[:n], pts[:n], keep_carry=True) if n else None for n in edges}
    empty = run_device(own_ctx, curve, np.zeros((1, 32), np.uint8), pts[:1])[0].tobytes()
    for i, n in enumerate(sizes):
        assert got[i].tobytes() == (want[n] if n else empty), n


@pytest.mark.parametrize("curve", [0, 1])
def test_batch_of_larger(own_ctx, large, curve):
    sizes = [7001, 24001, 90001, 150000]
    s, p = large[curve]
    n = sum(sizes)
    want = at_width(own_ctx, curve, 11, lambda: run_device(own_ctx, curve, s[:n], p[:n], sizes))
    assert (run_device(own_ctx, curve, s[:n], p[:n], sizes) == want).all()
