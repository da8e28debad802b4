"""2D sweeps as row strips and the parallel reflection points, at the sizes where their tiles,
strips and dispatch rules change: one row strip and many (32 rows each, 16 at most), a narrow last
column tile (64 columns each), grids too high or too wide for the strips in one precision or both,
more columns than the parallel reflection kernel takes, reflectors that fall one row per column
(each column waits for its neighbour).  Plain FP64: the oracle's bits, also where the iteration
limit ends the solve.  Mixed: the mode's bounds, 1e-5 for picks and 1e-4 for the gradient."""
import numpy as np
import pytest

from helpers import bits_equal

pytestmark = pytest.mark.gpu


def reflectors(n, nr, nc, d):
    """Depths with a flat part, then a slope of one row per column, then waves."""
    j = np.arange(nc)
    out = []
    for r in range(n):
        top = nr * (0.45 + 0.3 * r)
        z = top + np.minimum(np.maximum(j - nc // 3, 0), nr * 0.15) + 0.6 * np.sin(j / 5.0)
        out.append(np.stack([z * d, -np.ones(nc), np.zeros(nc)], 1))
    return np.concatenate(out) if n else None


@pytest.mark.parametrize("nr,nc,numofr,d,maxswp", [
    (3, 5, 0, (10.0, 10.0), 500), (32, 64, 1, (10.0, 10.0), 500), (33, 65, 2, (10.0, 10.0), 500),
    (31, 63, 1, (12.5, 8.3), 2), (64, 128, 1, (10.0, 10.0), 500), (97, 150, 2, (10.0, 5.0), 500),
    (97, 150, 2, (10.0, 10.0), 3), (512, 40, 1, (10.0, 10.0), 500), (513, 66, 1, (10.0, 10.0), 500),
    (500, 1000, 0, (10.0, 10.0), 500), (24, 5461, 1, (10.0, 10.0), 500), (24, 5462, 1, (10.0, 10.0), 500)])
def test_strips_and_reflection_points(ctx, nr, nc, numofr, d, maxswp):
    import torch
    import pfast_gb300 as pg
    from oracle import port
    dx, dz = d
    rng = np.random.default_rng(nr * 7 + nc)
    vp = 1500.0 + 8.0 * np.arange(nr)[:, None] + 300.0 * rng.random((nr, nc))
    Z = reflectors(numofr, nr, nc, dz)
    src = np.array([[0, nc // 5], [0, nc - 2], [min(nr - 1, 2), nc // 2]], np.int32)[:2 if nr * nc > 100000 else 3]
    rec1 = np.array([(0, j) for j in range(0, nc, max(1, nc // 60))], np.int32)
    rec = np.tile(rec1, (len(src), 1))
    srnum = np.full(len(src), len(rec1), np.int32)
    nxy = np.tile([-1.0, 0.0], (len(rec), 1))
    Tr0, _ = port.forward2d(vp, Z, src, srnum, rec, numofr, maxswp, dx, dz, nthreads=4)
    tt = Tr0[:, 0] + rng.normal(0, 1e-3, len(rec))
    tr = Tr0[:, 1:] + rng.normal(0, 1e-3, (len(rec), numofr))
    WR = np.full((nr, nc), 0.3)
    vp1 = vp * 1.02
    r0 = port.eval2d(vp1, WR, Z, src, srnum, rec, nxy, tt, tr, numofr, maxswp, dx, dz, nthreads=4)
    sv = pg.Survey2D(ctx, nr, nc, dx, dz, src, srnum, rec, numofr=numofr, Z=Z, nxy=nxy, tt_obs=tt,
                     tr_obs=tr if numofr else None)
    dvp, dvp1, dWR = (torch.from_numpy(a).cuda() for a in (vp, vp1, WR))
    Tr, _ = sv.forward(dvp, maxswp=maxswp)
    assert bits_equal(Tr.cpu().numpy(), Tr0)
    r = sv.eval(dvp1, dWR, maxswp=maxswp)
    for k in ("gT", "gR", "gRT"):
        assert bits_equal(r[k].cpu().numpy(), r0[k]), k
    assert r["Et"] == r0["Et"] and r["Er"] == r0["Er"]
    if maxswp == 500:
        Tm = sv.forward(dvp, precision=pg.PFAST_MIXED)[0].cpu().numpy()
        ok = Tr0 != 0
        assert np.max(np.abs(Tm - Tr0)[ok] / np.abs(Tr0[ok])) <= 1e-5
        g = sv.eval(dvp1, dWR, precision=pg.PFAST_MIXED)["gRT"].cpu().numpy()
        assert np.linalg.norm(g - r0["gRT"]) <= 1e-4 * np.linalg.norm(r0["gRT"])
    sv.close()
