"""Timed cases of the framework: the calls a traveltime-tomography user makes, with their
sizes, inputs, minimal work and 64-bit expectations.

listed() gives the named cases, draw(rng) one more of the same ranges, prepare(case, seed) the
state a user's program holds before the call (survey, model, picks), run(state) one pass through
the public entry points, work(case) the bytes and operations the pass cannot do without, and
exact(case, seed) the outputs as plain torch / numpy computes them in 64 bits: the fixed point
of the Godunov scheme and of the adjoint equation, to rounding.

The inputs are synthetic and seeded: a linear velocity gradient with a smooth +-5 % anomaly
field, sources and receivers near the surface, picks from the analytic traveltime of the
gradient medium (2D reflections: the image source) with 2 ms noise.
"""
import math

import numpy as np
import torch

import pfast_gb300 as pg

INF = 9999999.0        # unreached traveltime
MAXSWP3, MAXSWP2 = 100, 500

# ------------------------------------------------------------------ the cases


def listed():
    return [
        # the smallest call: one shot on a small odd grid through the reference-signature host function
        dict(name="solve3d_small", what="solve3d", nz=29, nr=37, nc=45, dx=20.0, dy=20.0, dz=20.0, nsrc=1),
        # one shot on an ordinary grid through the same function (a driver that calls source by source)
        dict(name="solve3d_one", what="solve3d", nz=64, nr=128, nc=128, dx=20.0, dy=20.0, dz=20.0, nsrc=1),
        # misfit and gradient in the default precision: a small 3D survey of an inversion run
        dict(name="grad3d_plain", what="grad3d", nz=48, nr=96, nc=96, dx=20.0, dy=20.0, dz=20.0, nsrc=16, step=4,
             mixed=False),
        # forward modelling of a field survey: ragged grid, unequal spacings, mixed precision
        dict(name="fwd3d_aniso", what="fwd3d", nz=101, nr=75, nc=155, dx=25.0, dy=20.0, dz=12.5, nsrc=24, step=3,
             mixed=True),
        # gradient of a 64-shot survey, mixed precision: few sources per SM
        dict(name="grad3d_mixed", what="grad3d", nz=64, nr=128, nc=128, dx=20.0, dy=20.0, dz=20.0, nsrc=64, step=4,
             mixed=True),
        # the headline workload: 256 x 256 x 128 nodes, 256 sources, 4096 receivers each
        dict(name="grad3d_large", what="grad3d", nz=128, nr=256, nc=256, dx=20.0, dy=20.0, dz=20.0, nsrc=256, step=4,
             mixed=True),
        # many independent models of uneven grids in one evaluation
        dict(name="many3d_mixed", what="many3d", models=8, nlo=200000, nhi=900000, slo=4, shi=40, mixed=True),
        # the one-call host-buffer form on a small odd survey: copies and survey set-up included
        dict(name="host3d_mixed", what="host3d", nz=53, nr=71, nc=90, dx=15.0, dy=20.0, dz=10.0, nsrc=9, step=5,
             mixed=True),
        # 2D first arrivals in the default precision (301 x 101 nodes, 21 shots)
        dict(name="fwd2d_plain", what="fwd2d", nr=101, nc=301, dx=10.0, dz=10.0, nsrc=21, step=2, refl=0, mixed=False),
        # 2D joint transmission + reflection gradient, mixed precision (601 x 201 nodes, 40 shots)
        dict(name="grad2d_mixed", what="grad2d", nr=201, nc=601, dx=5.0, dz=5.0, nsrc=40, step=2, refl=1, mixed=True),
        # the same in the default precision with two reflectors and unequal spacings
        dict(name="grad2d_plain", what="grad2d", nr=160, nc=600, dx=10.0, dz=5.0, nsrc=28, step=3, refl=2, mixed=False),
        # a whole call: two iterations of the 2D joint inversion loop (gradient, regularisation, L-BFGS, line search)
        dict(name="invert2d_mixed", what="invert2d", nr=101, nc=301, dx=10.0, dz=10.0, nsrc=12, step=3, refl=1,
             mixed=True, iters=2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    what = rng.choice(["solve3d", "grad3d", "grad3d", "fwd3d", "many3d", "host3d", "fwd2d", "grad2d", "grad2d", "invert2d"])
    if what == "many3d":
        return dict(what=what, models=rng.randint(3, 12), nlo=int(_log(rng, 6e4, 3e5)), nhi=int(_log(rng, 4e5, 1.2e6)),
                    slo=rng.randint(1, 6), shi=rng.randint(8, 40), mixed=rng.random() < 0.7)
    if what in ("fwd2d", "grad2d", "invert2d"):
        h = rng.choice([5.0, 10.0, 12.5])
        c = dict(what=what, nr=int(_log(rng, 45, 260)), nc=int(_log(rng, 60, 700)), dx=h,
                 dz=rng.choice([h, h, h / 2, 8.3]), nsrc=int(_log(rng, 1, 56.9)), step=rng.randint(1, 4),
                 refl=rng.randint(1, 2) if what == "invert2d" else rng.randint(0, 2), mixed=rng.random() < 0.5)
        if what == "invert2d":
            c.update(nsrc=min(c["nsrc"], 20), nc=min(c["nc"], 400), iters=rng.randint(1, 2))
        return c
    h = rng.choice([10.0, 20.0, 25.0])
    iso = rng.random() < 0.6
    c = dict(what=what, nz=int(_log(rng, 18, 128)), nr=int(_log(rng, 24, 256)), nc=int(_log(rng, 24, 256)), dx=h,
             dy=h if iso else rng.choice([15.0, 20.0, 16.7]), dz=h if iso else rng.choice([8.0, 12.5, 20.0]))
    if what == "solve3d":
        c["nsrc"] = 1
        return c
    c["mixed"] = rng.random() < 0.6
    most = (2.5e8 if c["mixed"] else 4e7) / (c["nz"] * c["nr"] * c["nc"])
    c["nsrc"] = max(1, min(int(_log(rng, 1, 256.9)), int(most)))
    c["step"] = rng.randint(2, 6)
    return c


# ------------------------------------------------------------------ inputs (from the seed alone)


def _noise(shape, coarse, rng):
    """Smooth noise of about unit range: coarse uniform noise, linearly interpolated."""
    small = [max(2, -(-n // coarse) + 1) for n in shape]
    t = torch.from_numpy(rng.uniform(-1.0, 1.0, small))[None, None]
    mode = "trilinear" if len(shape) == 3 else "bilinear"
    return torch.nn.functional.interpolate(t, size=tuple(shape), mode=mode, align_corners=True)[0, 0].numpy()


def _gradient_time(dist2, za, zb, v0, g):
    """First-arrival time between depths za and zb at squared distance dist2 in v0 + g z."""
    va, vb = v0 + g * za, v0 + g * zb
    return np.arccosh(1.0 + g * g * dist2 / (2.0 * va * vb)) / g


def _inputs3(case, seed):
    nz, nr, nc = case["nz"], case["nr"], case["nc"]
    dx, dy, dz = case["dx"], case["dy"], case["dz"]
    rng = np.random.default_rng([seed, nz, nr, nc, case["nsrc"]])
    v0, g = 2000.0, 0.6
    z = (np.arange(nz) + 1.0) * dz
    vp = (v0 + g * z)[:, None, None] * (1.0 + 0.05 * _noise((nz, nr, nc), 10, rng))
    vp = np.ascontiguousarray(vp)
    nsrc = case["nsrc"]
    # sources on a jittered surface grid, as a survey lays them out
    side = int(math.ceil(math.sqrt(nsrc)))
    cells = [(a, b) for a in range(side) for b in range(side)][:nsrc]
    src = np.zeros((nsrc, 3), np.int32)
    for s, (a, b) in enumerate(cells):
        src[s, 0] = min(nr - 1, int((a + rng.uniform(0.2, 0.8)) * nr / side))
        src[s, 1] = min(nc - 1, int((b + rng.uniform(0.2, 0.8)) * nc / side))
        src[s, 2] = rng.integers(0, 3)
    out = dict(vp=vp, src=src)
    if "step" not in case:
        return out
    st = case["step"]
    ri, rj = np.meshgrid(np.arange(st // 2, nr, st), np.arange(st // 2, nc, st), indexing="ij")
    rec1 = np.stack([ri.ravel(), rj.ravel(), np.zeros(ri.size, int)], 1).astype(np.int32)
    rec = np.ascontiguousarray(np.tile(rec1, (nsrc, 1)))
    srnum = np.full(nsrc, len(rec1), np.int32)
    nxyz = np.ascontiguousarray(np.tile([[0.0, 0.0, -1.0]], (len(rec), 1)))
    at = np.repeat(src, len(rec1), axis=0)
    d2 = ((rec[:, 0] - at[:, 0]) * dy) ** 2 + ((rec[:, 1] - at[:, 1]) * dx) ** 2 + ((rec[:, 2] - at[:, 2]) * dz) ** 2
    t = _gradient_time(d2, (rec[:, 2] + 1) * dz, (at[:, 2] + 1) * dz, v0, g)
    t = t * (1.0 + 0.02 * rng.standard_normal(nsrc).repeat(len(rec1))) + rng.normal(0.0, 0.002, len(t))
    t[rng.random(len(t)) < 0.05] = 999.0   # rows without a pick
    out.update(rec=rec, srnum=srnum, nxyz=nxyz, tobs=t)
    return out


def _many(case):
    """The single-model cases of a many-model evaluation (their sizes belong to the case)."""
    rng = np.random.default_rng([case["models"], case["nlo"], case["nhi"]])
    out = []
    for m in range(case["models"]):
        n = math.exp(rng.uniform(math.log(case["nlo"]), math.log(case["nhi"])))
        nz = max(20, int(round((n / 4.0) ** (1.0 / 3.0))))
        side = max(40, int(round(math.sqrt(n / nz))))
        out.append(dict(what="grad3d", nz=nz, nr=side, nc=side + int(rng.integers(-3, 4)), dx=20.0, dy=20.0, dz=20.0,
                        nsrc=int(rng.integers(case["slo"], case["shi"] + 1)), step=4, mixed=case["mixed"]))
    return out


def _inputs2(case, seed):
    nr, nc, dx, dz, nsrc, R = case["nr"], case["nc"], case["dx"], case["dz"], case["nsrc"], case["refl"]
    rng = np.random.default_rng([seed, nr, nc, nsrc, R])
    v0, depth = 1800.0, nr * dz
    g = 2200.0 / depth
    z = (np.arange(nr) + 1.0) * dz
    x = (np.arange(nc) + 1.0) * dx
    vp = np.ascontiguousarray((v0 + g * z)[:, None] * (1.0 + 0.05 * _noise((nr, nc), 12, rng)))
    cols = np.unique(np.round(np.linspace(2, nc - 3, nsrc) + rng.uniform(-1, 1, nsrc)).astype(int)) if nsrc > 1 else \
        np.array([int(rng.integers(2, nc - 2))])
    src = np.stack([np.zeros(len(cols), int), cols], 1).astype(np.int32)
    rec1 = np.stack([np.zeros(len(range(0, nc, case["step"])), int), np.arange(0, nc, case["step"])], 1).astype(np.int32)
    rec = np.ascontiguousarray(np.tile(rec1, (len(src), 1)))
    srnum = np.full(len(src), len(rec1), np.int32)
    nxy = np.ascontiguousarray(np.tile([[-1.0, 0.0]], (len(rec), 1)))
    at = np.repeat(src, len(rec1), axis=0)
    off2 = ((rec[:, 1] - at[:, 1]) * dx) ** 2
    tt = _gradient_time(off2, dz, dz, v0, g) + rng.normal(0.0, 0.002, len(rec))
    tt[rng.random(len(tt)) < 0.05] = 999.0
    Z = np.zeros((0, 3))
    tr = np.zeros((len(rec), R))
    if R:
        Z = []
        for ir in range(R):
            d = depth * (0.6 + 0.25 * ir) + 0.04 * depth * np.sin(2 * np.pi * x / (0.4 * nc * dx) + rng.uniform(0, 6)) \
                + rng.normal(0.0, 0.2 * dz, nc)
            slope = np.gradient(d, dx)
            nrm = np.sqrt(1.0 + slope ** 2)
            Z.append(np.stack([d, -1.0 / nrm, slope / nrm], 1))
            mean = d.mean()
            tr[:, ir] = np.sqrt(off2 + 4 * mean * mean) / (v0 + 0.45 * g * mean) + rng.normal(0.0, 0.002, len(rec))
            tr[rng.random(len(rec)) < 0.05, ir] = 0.0
        Z = np.concatenate(Z)
    WR = np.clip(np.broadcast_to((z / depth)[:, None], (nr, nc)), 0.1, 0.9).copy()
    return dict(vp=vp, src=src, rec=rec, srnum=srnum, nxy=nxy, tt=tt, tr=tr, Z=np.ascontiguousarray(Z), WR=WR)


# ------------------------------------------------------------------ states and passes

_CTX = []


def _ctx():
    """One context for the program, as its users keep it (stream and work buffers)."""
    if not _CTX:
        _CTX.append(pg.Context(0))
    return _CTX[0]


def _prec(case):
    return pg.PFAST_MIXED if case["mixed"] else pg.PFAST_PLAIN_FP64


def _survey3(case, d, picks):
    return pg.Survey3D(_ctx(), case["nr"], case["nc"], case["nz"], case["dx"], case["dy"], case["dz"], d["src"],
                       d["srnum"], d["rec"], d["nxyz"] if picks else None, d["tobs"] if picks else None)


def _survey2(case, d, picks):
    R = case["refl"]
    return pg.Survey2D(_ctx(), case["nr"], case["nc"], case["dx"], case["dz"], d["src"], d["srnum"], d["rec"], numofr=R,
                       Z=d["Z"] if R else None, nxy=d["nxy"] if picks else None, tt_obs=d["tt"] if picks else None,
                       tr_obs=d["tr"] if picks and R else None)


def prepare(case, seed):
    what = case["what"]
    s = dict(case=case, what=what)
    if what == "many3d":
        one = _many(case)
        ds = [_inputs3(c, seed + 1000 + m) for m, c in enumerate(one)]
        s["surveys"] = [_survey3(c, d, True) for c, d in zip(one, ds)]
        s["vps"] = [torch.from_numpy(d["vp"]).cuda() for d in ds]
        return s
    if what in ("fwd2d", "grad2d", "invert2d"):
        d = _inputs2(case, seed)
        s["survey"] = _survey2(case, d, what != "fwd2d")
        if what == "invert2d":
            s["vp"], s["WR"] = d["vp"], d["WR"]
        else:
            s["vp"], s["WR"] = torch.from_numpy(d["vp"]).cuda(), torch.from_numpy(d["WR"]).cuda()
        return s
    d = _inputs3(case, seed)
    if what == "solve3d":
        s.update(d, U=np.empty_like(d["vp"]))
    elif what == "host3d":
        s.update(d)
    else:
        s["survey"] = _survey3(case, d, what == "grad3d")
        s["vp"] = torch.from_numpy(d["vp"]).cuda()
    return s


def run(s):
    case, what = s["case"], s["what"]
    if what == "solve3d":
        pg.fsm3d(s["vp"], s["U"], s["src"], 0, MAXSWP3, case["dx"], case["dy"], case["dz"], case["nr"], case["nc"],
                 case["nz"])
        return {"T": s["U"]}
    if what == "grad3d":
        grad, misfit, _ = s["survey"].eval(s["vp"], precision=_prec(case))
        return {"grad": grad, "misfit": misfit}
    if what == "fwd3d":
        picks, _ = s["survey"].forward(s["vp"], precision=_prec(case))
        return {"picks": picks}
    if what == "many3d":
        grads, misfits, _ = pg.eval3d_many(_ctx(), s["surveys"], s["vps"], precision=_prec(case))
        return {"grads": grads, "misfits": misfits}
    if what == "host3d":
        grad, misfit, _ = pg.eval3d_host(_ctx(), s["vp"], case["dx"], case["dy"], case["dz"], s["src"], s["srnum"],
                                         s["rec"], s["nxyz"], s["tobs"], precision=_prec(case))
        return {"grad": grad, "misfit": misfit}
    if what == "fwd2d":
        picks, _ = s["survey"].forward(s["vp"], precision=_prec(case))
        return {"picks": picks}
    if what == "grad2d":
        r = s["survey"].eval(s["vp"], s["WR"], precision=_prec(case))
        return {k: r[k] for k in ("gT", "gR", "gRT", "Et", "Er")}
    inv = pg.Inversion(s["survey"], s["vp"], WR=s["WR"], LM=5, nux=6 * case["dx"], nuz=4 * case["dz"],
                       precision=_prec(case), conv_tol=-1.0)
    reps = [inv.step() for _ in range(case["iters"])]
    out = {"vp": inv.get("vp"), "grad_raw": inv.get("grad_raw"), "grad": inv.get("grad"),
           "E": [float(r["E"]) for r in reps]}
    inv.close()
    return out


# ------------------------------------------------------------------ minimal work
# Per source and node: one Godunov update (three minima, the sort, one quadratic: about 30
# operations in 3D, 18 in 2D) and one adjoint update (about 30 / 20); inputs read once, outputs
# written once.


def work(case):
    what = case["what"]
    if what == "many3d":
        per = [work(c) for c in _many(case)]
        return {k: sum(w[k] for w in per) for k in ("bytes", "flops")}
    if what in ("fwd2d", "grad2d", "invert2d"):
        n, R, ns = case["nr"] * case["nc"], case["refl"], case["nsrc"]
        rows = ns * -(-case["nc"] // case["step"])
        solves = ns * (1 + 2 * R)
        if what == "fwd2d":
            return {"bytes": 8 * (n + rows * (1 + R)), "flops": 18 * n * solves}
        grad = {"bytes": 8 * (5 * n + rows * (1 + R)), "flops": n * (18 * solves + 20 * ns * (1 + R))}
        if what == "grad2d":
            return grad
        return {k: v * 2 * case["iters"] for k, v in grad.items()}   # a gradient and at least one trial each
    n, ns = case["nz"] * case["nr"] * case["nc"], case["nsrc"]
    if what == "solve3d":
        return {"bytes": 16 * n, "flops": 30 * n}
    rows = ns * len(range(case["step"] // 2, case["nr"], case["step"])) * len(range(case["step"] // 2, case["nc"], case["step"]))
    if what == "fwd3d":
        return {"bytes": 8 * n + 8 * rows, "flops": 30 * n * ns}
    return {"bytes": 16 * n + 20 * rows, "flops": 60 * n * ns}


# ------------------------------------------------------------------ the same in 64 bits, plain torch


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _shift(U, dim, by, fill):
    """Neighbour values along dim: U at index + by, `fill` outside."""
    out = torch.full_like(U, fill)
    n = U.shape[dim]
    if by > 0:
        out.narrow(dim, 0, n - 1).copy_(U.narrow(dim, 1, n - 1))
    else:
        out.narrow(dim, 1, n - 1).copy_(U.narrow(dim, 0, n - 1))
    return out


def _axis_min(U, dim):
    return torch.minimum(_shift(U, dim, 1, math.inf), _shift(U, dim, -1, math.inf))


def _godunov(mins, hs, s):
    """Solution of sum_a (max(q - m_a, 0) / h_a)^2 = s^2 (any number of axes, unequal spacings),
    in difference form from the smallest minimum."""
    ms = list(mins)
    ws = [torch.full_like(ms[0], 1.0 / (h * h)) for h in hs]
    for a in range(len(ms)):   # ascending order of the minima, weights along
        for b in range(len(ms) - 1 - a):
            sw = ms[b] > ms[b + 1]
            ms[b], ms[b + 1] = torch.where(sw, ms[b + 1], ms[b]), torch.where(sw, ms[b], ms[b + 1])
            ws[b], ws[b + 1] = torch.where(sw, ws[b + 1], ws[b]), torch.where(sw, ws[b], ws[b + 1])
    s2 = s * s
    base = ms[0]
    q = base + s / torch.sqrt(ws[0])
    W, P, Q = ws[0].clone(), torch.zeros_like(base), torch.zeros_like(base)
    for a in range(1, len(ms)):
        d = ms[a] - base
        use = torch.isfinite(d) & (q > ms[a])
        d = torch.where(use, d, torch.zeros_like(d))
        W2, P2, Q2 = W + ws[a], P + ws[a] * d, Q + ws[a] * d * d
        # W x^2 - 2 P x + Q = s^2 with x = q - base
        D = P2 * P2 - W2 * (Q2 - s2)
        cand = base + (P2 + torch.sqrt(torch.clamp(D, min=0.0))) / W2
        q = torch.where(use, cand, q)
        W, P, Q = torch.where(use, W2, W), torch.where(use, P2, P), torch.where(use, Q2, Q)
    return q


def _solve(U, s, hs, dims, free):
    """Fixed point of U = min(U, Godunov(U)) on the nodes of `free`, in place."""
    for it in range(40 * sum(U.shape[d] for d in dims)):
        q = _godunov([_axis_min(U, d) for d in dims], hs, s)
        new = torch.where(free, torch.minimum(U, q), U)
        if it % 16 == 15 and float((U - new).max()) <= 1e-15:
            return new
        U = new
    return U


def _adjoint(lam, T, ws, dims, free):
    """Fixed point of lambda = num / den on the nodes of `free` (weights ws = 1 / h^2 per axis)."""
    reached = T < INF
    den, parts = torch.zeros_like(T), []
    for d, w in zip(dims, ws):
        for by in (1, -1):
            Tn = _shift(T, d, by, INF)
            reached &= Tn < INF
            e = Tn - T
            den += w * torch.clamp(-e, min=0.0)
            parts.append((d, by, w * torch.clamp(e, min=0.0)))
    ok = free & reached & (den > 1e-9)
    dead = free & ~ok
    coef = [(d, by, torch.where(ok, c / torch.where(ok, den, torch.ones_like(den)), torch.zeros_like(c))) for d, by, c in parts]
    lam = torch.where(dead, torch.zeros_like(lam), lam)
    keep = torch.where(free, torch.zeros_like(lam), lam)
    for it in range(40 * sum(T.shape[d] for d in dims)):
        new = keep.clone()
        for d, by, c in coef:
            new += c * _shift(lam, d, by, 0.0)
        if it % 16 == 15 and float((lam - new).abs().max()) <= 1e-15 * (1.0 + float(new.abs().max())):
            return new
        lam = new
    return lam


def _interior(shape, dims, dev):
    m = torch.ones(shape, dtype=torch.bool, device=dev)
    for d in dims:
        n = shape[d]
        m.narrow(d, 0, 1).fill_(False)
        m.narrow(d, n - 1, 1).fill_(False)
    return m


def _forward3(case, d, lo, hi, dev):
    shape = (hi - lo, case["nz"], case["nr"], case["nc"])
    U = torch.full(shape, INF, dtype=torch.float64, device=dev)
    free = torch.ones(shape, dtype=torch.bool, device=dev)
    for b in range(lo, hi):
        i, j, k = (int(v) for v in d["src"][b])
        U[b - lo, k, i, j] = 0.0
        free[b - lo, k, i, j] = False
    s = (1.0 / torch.from_numpy(d["vp"]).to(dev)).expand(shape)
    return _solve(U, s, (case["dx"], case["dy"], case["dz"]), (3, 2, 1), free)


def _exact3(case, seed, want_grad):
    d = _inputs3(case, seed)
    dev = _dev()
    n = case["nz"] * case["nr"] * case["nc"]
    chunk = max(1, int(6e7 // n))
    vp = torch.from_numpy(d["vp"]).to(dev)
    lamsum, E, picks = torch.zeros_like(vp), 0.0, []
    nr1 = len(d["rec"]) // case["nsrc"]
    for lo in range(0, case["nsrc"], chunk):
        hi = min(case["nsrc"], lo + chunk)
        T = _forward3(case, d, lo, hi, dev)
        rows = slice(lo * nr1, hi * nr1)
        rec = torch.from_numpy(d["rec"][rows].astype(np.int64)).to(dev)
        b = torch.arange(hi - lo, device=dev).repeat_interleave(nr1)
        i, j, k = rec[:, 0], rec[:, 1], rec[:, 2]
        t0 = T[b, k, i, j]
        if not want_grad:
            picks.append(t0)
            continue
        tob = torch.from_numpy(d["tobs"][rows]).to(dev)
        picked = tob < 100
        E += float((((tob - t0) ** 2) / 2.0)[picked].sum())

        def slope(axis_idx, size, h, at):
            up = axis_idx + 1 < size
            return torch.where(up, at(torch.where(up, axis_idx + 1, axis_idx)) - t0,
                               t0 - at(torch.where(up, axis_idx, axis_idx - 1))) / h
        Tz = slope(k, case["nz"], case["dz"], lambda q: T[b, q, i, j])
        Ty = slope(i, case["nr"], case["dy"], lambda q: T[b, k, q, j])
        Tx = slope(j, case["nc"], case["dx"], lambda q: T[b, k, i, q])
        nv = torch.from_numpy(d["nxyz"][rows]).to(dev)
        flux = nv[:, 1] * Tx + nv[:, 0] * Ty + nv[:, 2] * Tz
        v = torch.where(((tob - t0).abs() > 1e-9) & (flux.abs() > 1e-6), (tob - t0) / flux, torch.zeros_like(t0))
        src = torch.from_numpy(d["src"][lo:hi].astype(np.int64)).to(dev)[b]
        v = torch.where((src[:, 0] == i) & (src[:, 1] == j) & (src[:, 2] == k), torch.zeros_like(v), v)
        lam = torch.zeros_like(T)
        free = _interior(T.shape, (1, 2, 3), dev)
        at = (b[picked], k[picked], i[picked], j[picked])
        lam[at] = v[picked]
        free[at] = False
        lam = _adjoint(lam, T, (1 / case["dx"] ** 2, 1 / case["dy"] ** 2, 1 / case["dz"] ** 2), (3, 2, 1), free)
        lamsum += lam.sum(0)
    if not want_grad:
        return {"picks": torch.cat(picks)}
    return {"grad": -lamsum / vp ** 3, "misfit": E}


def _reflector(case, Zr):
    """Per column: lowest row above the reflector, reflection row, row limit of the up-going
    solve and the x-difference used there (0 central, 1 backward, 2 forward)."""
    nr, nc, dz = case["nr"], case["nc"], case["dz"]
    z = Zr[:, 0]
    down, k2, lim, qx = (np.full(nc, -1) for _ in range(4))
    i = np.arange(nr)
    for j in range(nc):
        above = np.nonzero((i + 1) * dz <= z[j])[0]
        down[j] = above[-1] if len(above) else -1
        nb = [z[q] for q in (j - 1, j + 1) if 0 <= q < nc]
        kk = i[:-1]
        ok = ((kk + 1) * dz + dz <= z[j]) & np.logical_or.reduce([kk * dz + dz <= q for q in nb])
        kk = kk[ok]
        if z[j] > nr * dz:
            lim[j] = nr - 1
            continue
        k2[j] = lim[j] = kk[-1]
        if j == 0:
            qx[j] = 2
        elif j == nc - 1:
            qx[j] = 1
        else:
            lo, hi = (k2[j] * dz + dz <= z[q] for q in (j - 1, j + 1))
            qx[j] = 0 if lo and hi else (1 if lo else 2)
    return down, k2, lim, qx


def _forward2(case, d, dev):
    """[transmission, up-going fields of the reflectors], each [nsrc, nr, nc]."""
    nr, nc, dx, dz, R = case["nr"], case["nc"], case["dx"], case["dz"], case["refl"]
    src, ns = d["src"], len(d["src"])
    s = (1.0 / torch.from_numpy(d["vp"]).to(dev)).expand(ns, nr, nc)
    rows = torch.arange(nr, device=dev)[:, None]

    def point():
        U = torch.full((ns, nr, nc), INF, dtype=torch.float64, device=dev)
        free = torch.ones((ns, nr, nc), dtype=torch.bool, device=dev)
        for b, (i, j) in enumerate(src):
            U[b, int(i), int(j)] = 0.0
            free[b, int(i), int(j)] = False
        return U, free

    U, free = point()
    out = [_solve(U, s, (dx, dz), (2, 1), free)]
    for ir in range(R):
        Zr = d["Z"][ir * nc:(ir + 1) * nc]
        down, k2, lim, qx = _reflector(case, Zr)
        U, free = point()
        U = _solve(U, s, (dx, dz), (2, 1), free & (rows <= torch.from_numpy(down).to(dev)))
        F = U.cpu().numpy()
        for jj in list(range(1, nc - 1)) + [0, nc - 1]:   # each column reads what the ones before wrote
            k = k2[jj]
            if k < 0:
                continue
            u0 = F[:, k, jj].copy()
            if qx[jj] == 0:
                px = (F[:, k, jj + 1] - F[:, k, jj - 1]) / 2.0 / dx
            elif qx[jj] == 1:
                px = (u0 - F[:, k, jj - 1]) / dx
            else:
                px = (F[:, k, jj + 1] - u0) / dx
            pz = (F[:, k + 1, jj] - u0) / dz
            zd, nz_, nx_ = Zr[jj]
            rz = pz - 2 * (px * nx_ + pz * nz_) * nz_
            F[:, k + 1, jj] = u0 + pz * (zd - k * dz - dz) + rz * ((k + 1) * dz + dz - zd)
        U = torch.from_numpy(F).to(dev)
        up = (rows <= torch.from_numpy(lim).to(dev)).expand(ns, nr, nc)
        U = torch.where(up, torch.full_like(U, INF), U)
        out.append(_solve(U, s, (dx, dz), (2, 1), up))
    return out


def _exact2(case, seed, want_grad):
    d = _inputs2(case, seed)
    dev = _dev()
    nr, nc, dx, dz, R = case["nr"], case["nc"], case["dx"], case["dz"], case["refl"]
    fields = _forward2(case, d, dev)
    ns = len(d["src"])
    nr1 = len(d["rec"]) // ns
    rec = torch.from_numpy(d["rec"].astype(np.int64)).to(dev)
    b = torch.arange(ns, device=dev).repeat_interleave(nr1)
    i, j = rec[:, 0], rec[:, 1]
    if not want_grad:
        return {"picks": torch.stack([F[b, i, j] for F in fields], 1)}
    src = torch.from_numpy(d["src"].astype(np.int64)).to(dev)[b]
    nv = torch.from_numpy(d["nxy"]).to(dev)
    vp = torch.from_numpy(d["vp"]).to(dev)
    sums, E, once = [torch.zeros_like(vp), torch.zeros_like(vp)], [0.0, 0.0], None
    for f, T in enumerate(fields):
        tob = torch.from_numpy(d["tt"] if f == 0 else d["tr"][:, f - 1]).to(dev)
        picked = tob < 100 if f == 0 else tob != 0
        t0 = T[b, i, j]
        E[f > 0] += float((((tob - t0) ** 2) / 2.0)[picked].sum())
        Tz = (T[b, i + 1, j] - t0) / dz   # receivers on the surface row
        right = j + 1 < nc
        Tx = torch.where(right, T[b, i, torch.where(right, j + 1, j)] - t0, t0 - T[b, i, torch.where(right, j, j - 1)]) / dx
        flux = nv[:, 1] * Tx + nv[:, 0] * Tz
        v = torch.where(((tob - t0).abs() > 1e-9) & (flux.abs() > 1e-6), (tob - t0) / flux, torch.zeros_like(t0))
        if f == 0:
            v = torch.where((src[:, 0] == i) & (src[:, 1] == j), torch.zeros_like(v), v)
        lam = torch.zeros_like(T)
        if f < 2:   # the reflectors of a source share one receiver mask
            once = _interior(T.shape, (1, 2), dev)
        at = (b[picked], i[picked], j[picked])
        lam[at] = v[picked]
        once[at] = False
        lam = _adjoint(lam, T, (1 / dx ** 2, 1 / dz ** 2), (2, 1), once)
        sums[f > 0] += lam.sum(0)
    gT, gR = (-x / vp ** 3 for x in sums)
    WR = torch.from_numpy(d["WR"]).to(dev)
    return {"gT": gT, "gR": gR, "gRT": gT * (1 - WR) + gR * WR, "Et": E[0], "Er": E[1]}


def exact(case, seed):
    what = case["what"]
    if what == "invert2d":
        return None   # its line search takes decisions; the gradients it is made of are cases of their own
    if what == "many3d":
        one = _many(case)
        r = [_exact3(c, seed + 1000 + m, True) for m, c in enumerate(one)]
        return {"grads": [x["grad"] for x in r], "misfits": [x["misfit"] for x in r]}
    if what in ("fwd2d", "grad2d"):
        return _exact2(case, seed, what == "grad2d")
    n = case["nz"] * case["nr"] * case["nc"]
    if n * case["nsrc"] * (case["nz"] + case["nr"] + case["nc"]) > 1.2e11:
        return None   # over 20 seconds
    if what == "solve3d":
        return {"T": _forward3(case, _inputs3(case, seed), 0, 1, _dev())[0]}
    return _exact3(case, seed, what != "fwd3d")
