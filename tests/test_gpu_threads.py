"""Evaluations of several threads at the same time, a context each: the 3D sweeps share the SMs among all
evaluations under way in the process (fewer blocks per source), which must not change a bit, nor the
iteration counts, against the same calls one after another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make3d(pg, ctx, shape, d, nsrc, seed):
    import torch
    nz, nr, nc = shape
    rng = np.random.default_rng(seed)
    vp = torch.from_numpy(1500.0 + 2500.0 * rng.random(shape)).cuda()
    src = np.stack([rng.integers(0, n, nsrc) for n in (nr, nc, nz)], 1).astype(np.int32)
    rec1 = np.array([(i, j, 0) for i in range(0, nr, 4) for j in range(0, nc, 5)], np.int32)
    rec = np.tile(rec1, (nsrc, 1))
    srnum = np.full(nsrc, len(rec1), np.int32)
    sv = pg.Survey3D(ctx, nr, nc, nz, *d, src, srnum, rec)
    vp1 = vp * 1.03
    torch.cuda.synchronize()
    tobs = sv.forward(vp1)[0].cpu().numpy()
    sv.close()
    sv = pg.Survey3D(ctx, nr, nc, nz, *d, src, srnum, rec, np.tile([0.0, 0.0, -1.0], (len(rec), 1)), tobs)

    def run(precision):
        g, e, s = sv.eval(vp, precision=precision)
        return [g.cpu().numpy().view(np.int64), e, s["fwd_iters_max"], s["adj_iters_max"], s["not_converged"]]
    return sv, run


def make2d(pg, ctx, seed):
    import torch
    nr, nc, n = 90, 150, 4
    rng = np.random.default_rng(seed)
    vp = torch.from_numpy(1500.0 + 8.0 * np.arange(nr)[:, None] + 300.0 * rng.random((nr, nc))).cuda()
    src = np.array([[0, j] for j in np.linspace(5, nc - 6, n).astype(int)], np.int32)
    rec1 = np.array([(0, j) for j in range(0, nc, 3)], np.int32)
    rec, srnum = np.tile(rec1, (n, 1)), np.full(n, len(rec1), np.int32)
    sv = pg.Survey2D(ctx, nr, nc, 10.0, 10.0, src, srnum, rec)
    vp1, wr = vp * 1.02, torch.zeros_like(vp)
    torch.cuda.synchronize()
    tt = sv.forward(vp1)[0].cpu().numpy()[:, 0]
    sv.close()
    sv = pg.Survey2D(ctx, nr, nc, 10.0, 10.0, src, srnum, rec, nxy=np.tile([-1.0, 0.0], (len(rec), 1)), tt_obs=tt)

    def run(precision):
        r = sv.eval(vp, wr, precision=precision)
        return [r["gT"].cpu().numpy().view(np.int64), r["Et"]]
    return sv, run


@pytest.mark.parametrize("nthreads", [2, 4])
def test_evaluations_of_several_threads(nthreads):
    import pfast_gb300 as pg
    kinds = [((16, 33, 64), (20.0, 20.0, 20.0), 9), None, ((21, 41, 70), (16.7, 12.5, 20.0), 30), ((12, 24, 96), (20.0, 20.0, 20.0), 1)]
    ctxs = [pg.Context(0) for _ in range(nthreads)]
    made = [make2d(pg, c, k) if kinds[k] is None else make3d(pg, c, *kinds[k], k) for k, c in enumerate(ctxs)]
    modes = (pg.PFAST_PLAIN_FP64, pg.PFAST_MIXED)
    want = [[run(m) for m in modes] for _, run in made]
    errors = []

    def work(k):
        try:
            for _ in range(4):
                for m, w in zip(modes, want[k]):
                    got = made[k][1](m)
                    for a, b in zip(got, w):
                        assert np.array_equal(a, b), (k, m)
        except BaseException as e:   # reported by the test's thread
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(nthreads)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (sv, _), c in zip(made, ctxs):
        sv.close()
        c.close()
    assert not errors, errors
