"""The forms of the polish kernels in the dataflow schedule that large surveys launch (kernels3d_tiles.cuh:
dataflow_form), with the bits of one launch per tile diagonal, on ragged grids with and without
aligned rows, in both tile shapes, and in one launch over several grids: the forward polish in
register windows (one block per source, 4096 tiles and more), the adjoint polish in windows in a
cluster (2 or 3 blocks per source, 1024 tiles and more)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ITERS = ("fwd_iters_max", "adj_iters_max", "fwd32_iters_max", "adj32_iters_max", "not_converged")


def survey(pg, ctx, shape, d, nsrc, seed):
    import torch
    nz, nr, nc = shape
    rng = np.random.default_rng(seed)
    z = np.arange(nz)[:, None, None] * d[2]
    vp = torch.from_numpy((2000.0 + 0.6 * z) * (1.0 + 0.05 * rng.standard_normal(shape).clip(-3, 3))).cuda()
    src = np.stack([rng.integers(0, n, nsrc) for n in (nr, nc, nz)], 1).astype(np.int32)
    rec1 = np.array([(i, j, 0) for i in range(0, nr, 9) for j in range(0, nc, 11)], np.int32)
    rec = np.tile(rec1, (nsrc, 1))
    srnum = np.full(nsrc, len(rec1), np.int32)
    sv = pg.Survey3D(ctx, nr, nc, nz, *d, src, srnum, rec)
    vp1 = vp * 1.02
    torch.cuda.synchronize()
    tobs = sv.forward(vp1, precision=pg.PFAST_MIXED)[0].cpu().numpy()
    sv.close()
    return vp, pg.Survey3D(ctx, nr, nc, nz, *d, src, srnum, rec, np.tile([0.0, 0.0, -1.0], (len(rec), 1)), tobs)


CASES = [
    ((66, 130, 472), (20.0, 20.0, 20.0), 110),    # forward windows, aligned rows
    ((65, 131, 469), (20.0, 25.0, 15.0), 105),    # the same, unaligned rows, unequal spacings
    ((46, 90, 300), (20.0, 20.0, 20.0), 60),      # adjoint windows in clusters of 3
    ((45, 91, 301), (12.5, 20.0, 20.0), 90),      # of 2, unaligned rows
]


@pytest.mark.parametrize("shape,d,nsrc", CASES)
@pytest.mark.parametrize("tile", [1, 2])
def test_polish_forms_same_bits(ctx, shape, d, nsrc, tile):
    import torch
    import pfast_gb300 as pg
    vp, sv = survey(pg, ctx, shape, d, nsrc, nsrc)
    g1, e1, s1 = sv.eval(vp, precision=pg.PFAST_MIXED, schedule=1, tile_shape=tile)
    for sched in (2, 3):
        g, e, s = sv.eval(vp, precision=pg.PFAST_MIXED, schedule=sched, tile_shape=tile)
        assert torch.equal(g.view(torch.int64), g1.view(torch.int64)) and e == e1
        assert all(s[k] == s1[k] for k in ITERS)
    sv.close()


@pytest.mark.parametrize("first,second", [(0, 1), (2, 3)])
def test_polish_forms_same_bits_in_one_launch(ctx, first, second):
    import torch
    import pfast_gb300 as pg
    cases = [(CASES[first][0], CASES[first][1], CASES[first][2] // 2), (CASES[second][0], CASES[second][1], CASES[second][2] // 2)]
    made = [survey(pg, ctx, *c, 7 + k) for k, c in enumerate(cases)]
    want = [sv.eval(vp, precision=pg.PFAST_MIXED, schedule=1, tile_shape=1)[:2] for vp, sv in made]
    grads, misfits = pg.eval3d_many(ctx, [sv for _, sv in made], [vp for vp, _ in made], precision=pg.PFAST_MIXED)[:2]
    for g, e, (g1, e1) in zip(grads, misfits, want):
        assert torch.equal(g.view(torch.int64), g1.view(torch.int64)) and e == e1
    for _, sv in made:
        sv.close()
