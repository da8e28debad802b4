"""The plain FP64 updates (pfast_gb300/csrc/exact_arith.h) outside the range of a survey's values: on the
CPU against the reference's expressions (tests/native/exact_range_check.cpp), and whole solves on the
GPU against the oracle, bit for bit (NaN for NaN): forward around bodies of almost no velocity (any
positive finite velocity is accepted), adjoint on fields with traveltimes that are no numbers,
infinite or huge (a caller's field is taken as it is)."""
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


@pytest.mark.parametrize("name", ["eik3_slowness", "eik2_slowness", "adj_axis_any_time", "adj_marking", "fwd_marking"])
def test_updates_match_the_expressions(check_lines, name):
    line = [x for x in check_lines if x.split()[1] == name]
    assert line and line[0].startswith("ok "), check_lines


# velocities whose slowness is on either side of 2^58, squares to infinity, to just below it, and is itself
# infinite
SLOW = [1e-9, 4e-18, 3e-18, 1e-60, 1e-130, 1e-140, 1e-152, 1e-160, 1e-300, 5e-324]


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


def same_or_nan(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    n = np.isnan(a)
    return np.array_equal(n, np.isnan(b)) and bits_equal(np.where(n, 0.0, a), np.where(n, 0.0, b))


@pytest.mark.gpu
@pytest.mark.parametrize("v", [np.nan, -np.nan, -np.inf, -1.7e308])
def test_adjoints_of_fields_with_any_time(v):
    import pfast_gb300 as pg
    from oracle import port
    rng = np.random.default_rng(11)
    nz, nr, nc = 6, 13, 40
    T = rng.uniform(0.0, 1.0, (nz, nr, nc))
    at = rng.random(T.shape) < 0.01
    at[0] = False                         # the receivers' plane keeps its times
    T[0] += 1.0                           # lambda enters from the receivers
    T[at] = v
    assert np.signbit(T[at]).all() == np.signbit(v) and at.sum() > 10
    src = np.array([[0, nc // 2, 0]], np.int32)
    rec = np.array([(i, j, 0) for i in range(nr) for j in range(nc)], np.int32)
    srnum = np.array([len(rec)], np.int32)
    n3 = np.tile([0.3, 0.1, -0.9], (len(rec), 1))
    tobs = T[0].ravel() + rng.normal(0.0, 0.02, len(rec))
    for d in ((20.0, 20.0, 20.0), (16.7, 8.3, 12.5)):
        L0, e0, _ = port.adjoint3d(T, tobs, rec, n3, src, srnum, 0, 40, *d)
        L = np.empty(T.shape)
        e = pg.adjoint_fsm3d(L, T, tobs, rec, n3, src, srnum, 0, 40, *d, nr, nc, nz)
        assert same_or_nan(L, L0) and e == e0
    T2 = np.ascontiguousarray(np.concatenate([T[0, :1], T[1], T[2], T[3]]))
    rec, n2, tobs, srnum, src = rec[:nc, :2].copy(), n3[:nc, :2].copy(), tobs[:nc].copy(), np.array([nc], np.int32), src[:, :2].copy()
    L0, e0, _ = port.tadjoint2d(T2, tobs, rec, n2, src, srnum, 0, 40, 20.0, 16.7)
    L = np.empty(T2.shape)
    e = pg.Tadjoint_fsm2d(L, T2, tobs, rec, n2, src, srnum, 0, 40, 20.0, 16.7, *T2.shape)
    assert same_or_nan(L, L0) and e == e0


@pytest.mark.gpu
@pytest.mark.parametrize("d,v0,contrast", [((19000.0, 17.5, 0.0027), 1e-175, 1.0), ((0.0027, 17.5, 19000.0), 1e-175, 1.0),
                                           ((20.0, 20.0, 20.0), None, 1e8), ((5.0, 100.0, 20.0), None, 1e6)])
def test_solves_far_from_the_source_in_steps(d, v0, contrast):
    """Uneven spacings and contrasts at which times are 1e7 steps and more: which tiles are skipped must
    still not show in the bits."""
    import pfast_gb300 as pg
    from oracle import port
    rng = np.random.default_rng(941)
    shape = nz, nr, nc = 36, 30, 41
    vp = 1500.0 + 2500.0 * rng.random(shape) if v0 else 1000.0 * np.exp(rng.uniform(0.0, np.log(contrast), shape))
    if v0:
        vp[rng.random(shape) < 0.05] = v0
    else:
        vp[rng.random(shape) < 0.3] = 1.0     # slow bodies around fast nodes
    src = np.stack([rng.integers(0, n, 20) for n in (nr, nc, nz)], 1).astype(np.int32)
    for s in range(len(src)):
        U0, _ = port.fsm3d(vp, src, s, 100, *d)
        U = np.empty_like(vp)
        pg.fsm3d(vp, U, src, s, 100, *d, nr, nc, nz)
        assert bits_equal(U, U0), s
