"""Mixed traveltimes of 1e-18 s and less (any positive finite velocity is accepted): the FP32 bulk sweeps
work with squares of a node's step there that are below the smallest normal FP32 number.  Velocities
scaled by a power of two scale every step of the bulk exactly until then (the polish drops corrections
below its floor of 1e-10 s, so it does nothing at either scale).  With steps sh of about 2^-66 the
discriminants are rounded to 2^-149, which is at most 2^-74.5 / 2^-65.5 = 2e-3 of a step in each step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_bulk_sweeps_of_tiny_times(ctx):
    import torch
    import pfast_gb300 as pg
    rng = np.random.default_rng(3)
    nz, nr, nc, h = 12, 30, 40, 20.0
    vp = rng.uniform(1500.0, 2500.0, (nz, nr, nc))
    src = np.array([[3, 4, 1], [20, 30, 8]], np.int32)
    rec1 = np.array([(i, j, 0) for i in range(0, nr, 3) for j in range(0, nc, 3)], np.int32)
    rec, srnum = np.tile(rec1, (2, 1)), np.full(2, len(rec1), np.int32)
    sv = pg.Survey3D(ctx, nr, nc, nz, h, h, h, src, srnum, rec)
    out = []
    for k in (33, 59):
        p, st = sv.forward(torch.from_numpy(vp * 2.0 ** k).cuda(), precision=pg.PFAST_MIXED)
        assert st["not_converged"] == 0
        out.append(p.cpu().numpy() * 2.0 ** k)
    sv.close()
    assert out[0].min() > 0.0 and np.max(np.abs(out[1] / out[0] - 1.0)) <= 2e-3


def test_steps_on_both_sides_of_the_line(ctx):
    """Steps scaled by powers of two to just above 2^-37 s, just below it and far below (the line between the
    two forms of the square root): the bulk's times scale exactly, no correction reaching the polish floor."""
    import torch
    import pfast_gb300 as pg
    rng = np.random.default_rng(4)
    nz, nr, nc, h = 9, 21, 70, 20.0
    vp = rng.uniform(1500.0, 2500.0, (nz, nr, nc))
    vp[0, 0, 0] = 2500.0                       # the least step is 2^-6.97 s
    src = np.array([[3, 4, 1], [20, 30, 8]], np.int32)
    rec1 = np.array([(i, j, 0) for i in range(0, nr, 2) for j in range(0, nc, 3)], np.int32)
    rec, srnum = np.tile(rec1, (2, 1)), np.full(2, len(rec1), np.int32)
    sv = pg.Survey3D(ctx, nr, nc, nz, h, h, h, src, srnum, rec)
    out = {}
    for k in (24, 30, 31, 40):
        p, st = sv.forward(torch.from_numpy(vp * 2.0 ** k).cuda(), precision=pg.PFAST_MIXED, polish_floor=9e-10)
        out[k] = p.cpu().numpy() * 2.0 ** k
        assert st["not_converged"] == 0
    sv.close()
    assert all(np.array_equal(out[k], out[24]) for k in out)
