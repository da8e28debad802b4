"""The plain FP64 updates (pfast_gb300/csrc/exact_arith.h) outside the range of a survey's values: on the
CPU against the reference's expressions (tests/native/exact_range_check.cpp), and whole solves on the
GPU against the oracle, bit for bit, around bodies of almost no velocity (any positive finite
velocity is accepted)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import bits_equal

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def check_lines(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path_factory.mktemp("exact_range") / "check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "pfast_gb300", "csrc"),
                    os.path.join(HERE, "native", "exact_range_check.cpp"), "-o", exe], check=True)
    return subprocess.run([exe], capture_output=True, text=True, timeout=300).stdout.splitlines()


@pytest.mark.parametrize("name", ["eik3_slowness", "eik2_slowness"])
def test_updates_match_the_expressions(check_lines, name):
    line = [x for x in check_lines if x.split()[1] == name]
    assert line and line[0].startswith("ok "), check_lines


# velocities whose slowness squares to infinity, to just below it, and is itself infinite
SLOW = [1e-130, 1e-140, 1e-152, 1e-160, 1e-300, 5e-324]


@pytest.mark.gpu
@pytest.mark.parametrize("v0", SLOW)
def test_solves_around_impermeable_bodies(v0):
    import torch
    import pfast_gb300 as pg
    from oracle import port
    rng = np.random.default_rng(5)
    nz, nr, nc = 9, 21, 37
    vp = 1500.0 + 1000.0 * rng.random((nz, nr, nc))
    vp[2:6, 5:12, 8:20] = v0
    vp[rng.random(vp.shape) < 0.03] = v0
    src = np.array([[2, 3, 1]], np.int32)
    for d in ((20.0, 20.0, 20.0), (16.7, 8.3, 12.5)):
        U0, _ = port.fsm3d(vp, src, 0, 100, *d)
        U = np.empty_like(vp)
        pg.fsm3d(vp, U, src, 0, 100, *d, nr, nc, nz)
        assert np.isfinite(U0).all() and bits_equal(U, U0)
    vp2 = np.ascontiguousarray(np.concatenate(list(vp[:3])))
    rec = np.array([(i, j) for i in range(0, 3 * nr, 3) for j in range(0, nc, 2)], np.int32)
    srnum = np.array([len(rec)], np.int32)
    ctx = pg.Context(0)
    for dx, dz in ((20.0, 20.0), (16.7, 8.3)):
        Tr0, _ = port.forward2d(vp2, None, src[:, :2].copy(), srnum, rec, 0, 500, dx, dz)
        sv = pg.Survey2D(ctx, 3 * nr, nc, dx, dz, src[:, :2].copy(), srnum, rec)
        Tr, _ = sv.forward(torch.from_numpy(vp2).cuda())
        assert bits_equal(Tr.cpu().numpy(), Tr0)
        sv.close()
    ctx.close()
