"""The dataflow schedule with a thread-block cluster per source: the policy that picks the cluster
size and the untuned schedule (pfast_gb300/csrc/tune_policy.h, compiled with g++), and on the GPU
the same bits as one launch per tile diagonal for source counts that give clusters of 1 to 9
blocks and of the tile count's most, whole and ragged tiles, equal and unequal spacings."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHECK = r"""
#include <cstdio>
#include "tune_policy.h"
using namespace pfast;
static int n = 0;
static void eq(long long got, long long want) { ++n; std::printf("%s %d: %lld %lld\n", got == want ? "ok" : "FAIL", n, got, want); }
static int size(bool plain, int nact, int ntiles) {
    for (int cs = kMaxCluster; cs > 1; --cs) if (cluster_wanted(cs, plain, nact, ntiles, 152)) return cs;
    return 1;
}
int main() {
    eq(size(true, 1, 1024), 16); eq(size(true, 16, 432), 8); eq(size(true, 40, 432), 4); eq(size(true, 100, 432), 1);
    eq(size(false, 9, 378), 16); eq(size(false, 24, 1300), 8); eq(size(false, 64, 1024), 3); eq(size(false, 256, 8192), 1);
    eq(size(false, 1, 80), 8); eq(size(false, 1, 15), 1);
    eq(size(true, 21, 1600), 7); eq(size(true, 42, 432), 3); eq(size(true, 12, 432), 8); eq(size(true, 12, 1300), 13);
    for (int cs = 2; cs <= 16; cs *= 2) eq(cluster_warps(cs, true) >= 4 && cluster_warps(cs, false) <= 24, 1);
    // schedule: candidate 2 = dataflow 4x8x32, 0 = per diagonal 4x8x32
    eq(untuned_pick(0x3f, true, false, 16, 1, 1024, 34, 152), 2);
    eq(untuned_pick(0x3f, true, false, 1, 100, 432, 26, 152), 0);
    eq(untuned_pick(0x3f, true, false, 1, 200, 432, 26, 152), 2);
    eq(untuned_pick(0x3f, true, false, 1, 84, 128, 16, 152), 2);      // few tiles a diagonal
    eq(untuned_pick(0x3f, true, false, 2, 61, 680, 28, 152), 0);
    eq(untuned_pick(0x3f, true, false, 2, 79, 864, 43, 152), 2);
    eq(untuned_pick(0x3f, true, false, 7, 23, 1736, 44, 152), 2);
    eq(untuned_pick(0x3f, false, true, 1, 256, 8192, 70, 152), 0);
    eq(untuned_pick(0x3f, false, true, 1, 300, 1024, 34, 152), 2);
    eq(untuned_pick(0x3f, false, false, 1, 256, 8192, 70, 152), 2);
    eq(untuned_pick(0x03, false, false, 1, 256, 8192, 70, 152), 0);   // per diagonal asked for
    eq(untuned_pick(0x2a, false, false, 1, 256, 8192, 70, 152), 3);   // 8x4x32 asked for
    eq(untuned_pick(0x30, true, false, 1, 100, 432, 26, 152), 4);     // hybrid asked for
    TuneEntry e;
    eq(tune_complete(&e, 0x3f), 0); eq(tune_complete(nullptr, 1), 0);
    e.n[0] = e.n[2] = 1;
    eq(tune_complete(&e, 0x5), 1);
}
"""


def test_cluster_and_schedule_policy(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "check.cpp", str(tmp_path / "check")
    src.write_text(CHECK)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "pfast_gb300", "csrc"), str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout
    assert "FAIL" not in out and out.count("ok ") == 34, out


@pytest.mark.gpu
@pytest.mark.parametrize("shape,d,nsrc", [((16, 33, 64), (20.0, 20.0, 20.0), n) for n in (1, 30, 45, 170)] +
                         [((21, 41, 70), (16.7, 12.5, 20.0), n) for n in (1, 9, 22, 27, 60)] +
                         [((40, 72, 320), (20.0, 20.0, 20.0), 17)])
def test_cluster_dataflow_same_bits(shape, d, nsrc):
    import torch
    import pfast_gb300 as pg
    nz, nr, nc = shape
    rng = np.random.default_rng(nsrc + nc)
    vp = torch.from_numpy(1500.0 + 2500.0 * rng.random(shape)).cuda()
    src = np.stack([rng.integers(0, n, nsrc) for n in (nr, nc, nz)], 1).astype(np.int32)
    rec1 = np.array([(i, j, 0) for i in range(0, nr, 4) for j in range(0, nc, 5)], np.int32)
    rec = np.tile(rec1, (nsrc, 1))
    srnum = np.full(nsrc, len(rec1), np.int32)
    nxyz = np.tile([0.0, 0.0, -1.0], (len(rec), 1))
    ctx = pg.Context(0)
    sv = pg.Survey3D(ctx, nr, nc, nz, *d, src, srnum, rec)
    tobs = sv.forward(vp * 1.03)[0].cpu().numpy()
    sv.close()
    sv = pg.Survey3D(ctx, nr, nc, nz, *d, src, srnum, rec, nxyz, tobs)
    for prec in (pg.PFAST_PLAIN_FP64, pg.PFAST_MIXED):
        g1, e1, s1 = sv.eval(vp, precision=prec, schedule=1, tile_shape=1)
        for sched in (0, 2, 3):
            g, e, s = sv.eval(vp, precision=prec, schedule=sched, tile_shape=1)
            assert torch.equal(g.view(torch.int64), g1.view(torch.int64)) and e == e1
            assert all(s[k] == s1[k] for k in ("fwd_iters_max", "adj_iters_max", "fwd32_iters_max", "adj32_iters_max",
                                               "not_converged"))
    sv.close()
    ctx.close()
