"""The plain FP64 updates with fewer FP64 instructions (pfast_gb300/csrc/exact_arith.h): against the
reference's expressions as they stand on the CPU (tests/native/exact_arith_check.cpp: divisions by
constants, 3D / 2D Godunov updates and adjoint terms, random and edge arguments), and whole plain
solves on the GPU, whose tiles are skipped by dependency, against the oracle: rough models, long
and short spacings, the smallest grids.  Everything bit for bit."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_exact_updates_match_the_expressions(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "exact_arith_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "pfast_gb300", "csrc"),
                    os.path.join(HERE, "native", "exact_arith_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "FAIL" not in out.stdout and out.stdout.count("ok ") == 10, out.stdout


def _bits(a):
    return np.ascontiguousarray(a).view(np.int64)


@pytest.mark.gpu
@pytest.mark.parametrize("schedule", [1, 2, 3])
@pytest.mark.parametrize("shape,d,scale", [((2, 2, 2), (20.0, 20.0, 20.0), 1.0), ((5, 9, 33), (16.7, 8.3, 20.0), 1.0),
                                           ((13, 17, 66), (20.0, 20.0, 20.0), 1.0), ((8, 24, 31), (0.1, 0.3, 0.1), 1.0),
                                           ((6, 10, 34), (12.5, 12.5, 12.5), 1e250)])
def test_plain_solves_bitwise_rough_models(schedule, shape, d, scale):
    """scale 1e250: velocities beyond the range of the shortened updates (the expressions as they stand)."""
    import torch
    import pfast_gb300 as pg
    from oracle import port
    nz, nr, nc = shape
    rng = np.random.default_rng(nz * nr + nc)
    vp = np.exp(rng.uniform(np.log(500.0), np.log(8000.0), shape)) * scale
    src = np.array([[nr // 2, nc // 2, 0], [0, nc - 1, nz - 1]], np.int32)
    rec1 = np.array([(i, j, 0) for i in range(0, nr, 2) for j in range(0, nc, 3)], np.int32)
    rec = np.concatenate([rec1, rec1])
    srnum = np.full(2, len(rec1), np.int32)
    nxyz = np.tile([0.1, -0.2, -0.97], (len(rec), 1))
    dx, dy, dz = d
    pk = port.forward3d(vp, src, srnum, rec, 100, dx, dy, dz)
    tobs = pk + rng.normal(0.0, 0.01, len(pk)) * (1.0 if scale == 1.0 else 1e-3)
    g0, e0, _, _ = port.eval3d(vp, src, srnum, rec, nxyz, tobs, 100, dx, dy, dz)
    ctx = pg.Context(0)
    sv = pg.Survey3D(ctx, nr, nc, nz, dx, dy, dz, src, srnum, rec, nxyz, tobs)
    d_vp = torch.from_numpy(vp).cuda()
    p, _ = sv.forward(d_vp, schedule=schedule)
    assert np.array_equal(_bits(p.cpu().numpy()), _bits(pk))
    g, e, _ = sv.eval(d_vp, schedule=schedule)
    assert np.array_equal(_bits(g.cpu().numpy()), _bits(g0)) and e == e0
    sv.close()
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("shape,dx,dz", [((2, 2), 10.0, 10.0), ((33, 65), 16.7, 8.3), ((70, 140), 5.0, 5.0)])
def test_plain_adjoint_of_any_traveltime_field(shape, dx, dz):
    """The adjoints take the caller's traveltimes: negative, equal, unreached and rough ones."""
    import pfast_gb300 as pg
    from oracle import port
    nr, nc = shape
    rng = np.random.default_rng(nr + nc)
    for kind in range(3):
        T = rng.uniform(-1.0, 1.0, shape) if kind == 0 else np.round(rng.uniform(0.0, 1.0, shape), 1)
        if kind == 2:
            T[rng.random(shape) < 0.02] = 9999999.0
        src = np.array([[0, nc // 2]], np.int32)
        rec = np.array([(0, j) for j in range(nc)], np.int32)
        srnum = np.array([nc], np.int32)
        nxy = np.tile([-0.9, 0.3], (nc, 1))
        tobs = T[0] + rng.normal(0.0, 0.02, nc)
        tobs[::5] = 200.0
        L0, e0, _ = port.tadjoint2d(T, tobs, rec, nxy, src, srnum, 0, 40, dx, dz)
        L = np.empty(shape)
        e = pg.Tadjoint_fsm2d(L, T, tobs, rec, nxy, src, srnum, 0, 40, dx, dz, nr, nc)
        assert np.array_equal(_bits(L), _bits(L0)) and e == e0
        T3 = np.ascontiguousarray(np.stack([T, T + 0.01, T - 0.02, np.roll(T, 1)]))
        src3, rec3 = np.array([[0, nc // 2, 0]], np.int32), np.array([(0, j, 0) for j in range(nc)], np.int32)
        n3 = np.tile([0.3, 0.1, -0.9], (nc, 1))
        L0, e0, _ = port.adjoint3d(T3, tobs, rec3, n3, src3, srnum, 0, 40, dx, dx, dz)
        L = np.empty(T3.shape)
        e = pg.adjoint_fsm3d(L, T3, tobs, rec3, n3, src3, srnum, 0, 40, dx, dx, dz, nr, nc, 4)
        assert np.array_equal(_bits(L), _bits(L0)) and e == e0
