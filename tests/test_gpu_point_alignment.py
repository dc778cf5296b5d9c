"""Device points that start on a 16-byte but not a 32-byte boundary: the kernels
that load a coordinate at once where the points allow it give the same bytes as
for aligned points, in every accumulation form and at sizes around their
blocks."""

import numpy as np
import pytest

import helioselene_gb300 as hs
from conftest import oracle_inputs

pytestmark = pytest.mark.gpu


def shifted(torch, data: np.ndarray, offset: int):
    buf = torch.zeros(data.size + 64, dtype=torch.uint8, device="cuda:0")
    t = buf[offset:offset + data.size]
    t.copy_(torch.from_numpy(data.copy()))
    assert t.data_ptr() % 32 == offset % 32
    return t


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("n,rounds", [(1, 0), (37, 0), (3000, 0), (8192, 0), (2049, 1), (5000, 2), (4096, 3), (9001, 2)])
def test_msm_of_points_at_16_bytes(ctx, curve, n, rounds):
    torch = pytest.importorskip("torch")
    sc, pts, _ = oracle_inputs(curve, n, seed=n + rounds, edge_fraction=0.02)
    d_sc = torch.from_numpy(sc.reshape(-1).copy()).to("cuda:0")
    if rounds:
        ctx.set_batch_affine(rounds, 1, curve)
    try:
        got = []
        for offset in (0, 16):
            d_pts = shifted(torch, pts.reshape(-1), offset)
            out = torch.zeros(32, dtype=torch.uint8, device="cuda:0")
            torch.cuda.synchronize()
            ctx.msm_device(curve, d_sc.data_ptr(), d_pts.data_ptr(), n, out.data_ptr(), hs.FMT_COMPRESSED)
            torch.cuda.synchronize()
            got.append(out.cpu().numpy().tobytes())
    finally:
        ctx.default_batch_affine()
    import oracle
    assert got[0] == got[1] == oracle.msm(curve, sc, pts, keep_carry=True)


@pytest.mark.parametrize("curve", [0, 1])
def test_scalar_mul_of_points_at_16_bytes(ctx, curve):
    torch = pytest.importorskip("torch")
    sc, pts, _ = oracle_inputs(curve, 129, seed=5)
    d_sc = torch.from_numpy(sc.reshape(-1).copy()).to("cuda:0")
    got = []
    for offset in (0, 16):
        d_pts = shifted(torch, pts.reshape(-1), offset)
        out = torch.zeros(129 * 64, dtype=torch.uint8, device="cuda:0")
        torch.cuda.synchronize()
        ctx.scalar_mul_device(curve, d_sc.data_ptr(), d_pts.data_ptr(), 129, out.data_ptr(), hs.FMT_AFFINE)
        torch.cuda.synchronize()
        got.append(out.cpu().numpy().tobytes())
    assert got[0] == got[1]


@pytest.mark.parametrize("curve", [0, 1])
@pytest.mark.parametrize("offset", [0, 16])
def test_scalar_mul_of_points_at_16_bytes_against_the_oracle(ctx, curve, offset):
    torch = pytest.importorskip("torch")
    import oracle
    sc, pts, _ = oracle_inputs(curve, 33, seed=6)
    d_sc, d_pts = torch.from_numpy(sc.reshape(-1).copy()).to("cuda:0"), shifted(torch, pts.reshape(-1), offset)
    out = torch.zeros(33 * 32, dtype=torch.uint8, device="cuda:0")
    torch.cuda.synchronize()
    ctx.scalar_mul_device(curve, d_sc.data_ptr(), d_pts.data_ptr(), 33, out.data_ptr(), hs.FMT_COMPRESSED)
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(33, 32)
    for i in range(33):
        assert got[i].tobytes() == oracle.msm(curve, sc[i:i + 1], pts[i:i + 1]), i
