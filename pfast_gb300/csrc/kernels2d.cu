// kernels2d.cu -- 2D fast-sweeping Eikonal (with Huygens reflection) and adjoint
// kernels for sm_103a.
//
// Same scheme as the 3D kernels: the 4 sweep orders of the reference
// (src/RT_pfsm2d.h:168-181, src/RT_padjoint2d.h:351-369) are run as wavefronts of
// T2I x T2J tiles, with one launch per phase in which a warp streams along each strip of
// T2I rows (up to 512 rows; taller grids take one launch per tile anti-diagonal); lane =
// row, and step t updates the node anti-diagonal li + lj = t.  Upstream neighbours are
// final and downstream ones untouched when a node is updated, exactly as in the
// reference's lexicographic loop, so the plain FP64 flavour is bit-identical.

#include <vector>
#include <algorithm>
#include <type_traits>
#include "kernels2d.h"
#include "strip_sync.h"

namespace pfast {

namespace {

template <int KIND> struct Traits2;
template <> struct Traits2<kFwdPlain64>  { using Real = double; using Aux = double; static constexpr bool adj = false; };
template <> struct Traits2<kFwdFast32>   { using Real = float;  using Aux = float;  static constexpr bool adj = false; };
template <> struct Traits2<kFwdPolish64> { using Real = double; using Aux = double; static constexpr bool adj = false; };
template <> struct Traits2<kAdjPlain64>  { using Real = double; using Aux = double; static constexpr bool adj = true; };
template <> struct Traits2<kAdjFast32>   { using Real = float;  using Aux = float;  static constexpr bool adj = true; };
template <> struct Traits2<kAdjPolish64> { using Real = double; using Aux = double; static constexpr bool adj = true; };

// The FP64 adjoint kinds read the traveltime through register windows (no second FP64 box);
// the FP32 bulk adjoint stages it as a box of FP32 offsets.
template <int KIND>
__host__ __device__ constexpr bool t_windows2() {
    return Traits2<KIND>::adj && sizeof(typename Traits2<KIND>::Aux) == 8;
}

template <int KIND>
__host__ __device__ constexpr int warp_smem2() {
    using T = Traits2<KIND>;
    return int(H2I * R2 * sizeof(typename T::Real) +
               (T::adj && !t_windows2<KIND>() ? H2I * R2 * sizeof(typename T::Aux) : 0));
}

__device__ __forceinline__ double ref_min(double x, double y) { return min_nonneg(x, y); }   // values >= +0
__device__ __forceinline__ float ref_min(float x, float y) { return (x < y) ? x : y; }

// Reference 2D Godunov update (src/RT_pfsm2d.h:89-102), operand order kept (exact_arith.h, or
// for spacings outside its range the expressions as they stand).
// a: x-neighbour minimum (spacing dx), b: z-neighbour minimum (dz).
__device__ __forceinline__ double eik2_plain(double a, double b, double s, const Sweep2Args& K) {
    if (K.ex.quick) return K.ex.fast ? eik2_exact<true>(a, b, s, K.ex) : eik2_exact<false>(a, b, s, K.ex);
    double da = K.dx, db = K.dz, ia = K.inv2x, ib = K.inv2z, t;
    if (b > a) { t = a; a = b; b = t; t = da; da = db; db = t; t = ia; ia = ib; ib = t; }
    double q = b + db * s;
    if (q <= a) return q;
    const double A = ia + ib;   // 1.0/da/da + 1.0/db/db with each term precomputed as (1.0/d)/d
    const double B = -2. * (a / da / da + b / db / db);
    const double C = a * a / da / da + b * b / db / db - s * s;
    const double D = B * B - 4 * A * C;
    return (D >= 0) ? (-B + sqrt(D)) / 2. / A : kInf;
}

// Same solution in difference form: x = q - b, with B = a - b >= 0:
//   1 term  x = db*s;  2 terms  x = (wa*B + sqrt((wa+wb) s^2 - wa wb B^2)) / (wa+wb)
template <typename R>
__device__ __forceinline__ R eik2_fast(R a, R b, R s, R dx, R dz, R wx, R wz, R rsum) {
    R da = dx, db = dz, wa = wx, wb = wz, t;
    if (b > a) { t = a; a = b; b = t; t = da; da = db; db = t; t = wa; wa = wb; wb = t; }
    R q = fma(db, s, b);
    if (q <= a) return q;
    const R B = a - b;
    const R waB = wa * B;
    const R D = fma(wa + wb, s * s, -waB * wb * B);
    return (D >= R(0)) ? b + (waB + sqrt(D)) * rsum : R(kInf);
}

// The FP32 form without branches: in a step the lanes' nodes fall into both cases anyway (the
// same expressions, selected; a discriminant below 0 is never selected).
__device__ __forceinline__ float eik2_fast_sel(float a, float b, float s, float dx, float dz, float wx, float wz, float rsum) {
    const bool sw = b > a;
    const float hi = sw ? b : a, lo = sw ? a : b, dl = sw ? dx : dz, wh = sw ? wz : wx, wl = sw ? wx : wz;
    const float q = fmaf(dl, s, lo);
    const float B = hi - lo;
    const float wB = wh * B;
    const float D = fmaf(wh + wl, s * s, -wB * wl * B);
    const float r = (D >= 0.0f) ? lo + (wB + sqrtf(D)) * rsum : (float)kInf;
    return q <= hi ? q : r;
}

__device__ __forceinline__ double pos_ref(double x) { return (x + fabs(x)) / 2.0; }
__device__ __forceinline__ double neg_ref(double x) { return (x - fabs(x)) / 2.0; }

// Reference 2D adjoint update (src/RT_padjoint2d.h:42-65), as eik2_plain.
__device__ __forceinline__ double adj2_plain(double T0, double Txp, double Txm, double Tzp, double Tzm, double Lxp,
                                             double Lxm, double Lzp, double Lzm, const Sweep2Args& K) {
    const long long inf = dbits(kInf);   // T >= INF on the bit patterns (T >= 0)
    if (dbits(Txp) >= inf || dbits(T0) >= inf || dbits(Txm) >= inf || dbits(Tzp) >= inf || dbits(Tzm) >= inf)
        return 0.0;
    const unsigned most = most_of(most_of(upper_of(T0), upper_of(Txp)),
                                  most_of(upper_of(Txm), most_of(upper_of(Tzp), upper_of(Tzm))));
    if (K.ex.quick && adj_ordinary(most)) {
        double ex, ez, nx, nz;
        adj_axis_exact(T0, Txp, Txm, Lxp, Lxm, K.ex.x, ex, nx);
        adj_axis_exact(T0, Tzp, Tzm, Lzp, Lzm, K.ex.z, ez, nz);
        const double den = ex + ez;
        const double num = nx + nz;   // den >= 0: a zero keeps its sign, and needs no division (its slow path)
        return fabs(den) > 1e-9 ? (is_zero(num) ? num : here(num) / den) : 0.0;
    }
    const double dx = K.dx, dz = K.dz;
    const double gxp = -(Txp - T0) / dx, gxm = -(T0 - Txm) / dx;
    const double gzp = -(Tzp - T0) / dz, gzm = -(T0 - Tzm) / dz;
    const double a1 = pos_ref(gxp), a2 = neg_ref(gxm);
    const double b1 = pos_ref(gzp), b2 = neg_ref(gzm);
    const double La1 = pos_ref(gxm) * Lxm, La2 = neg_ref(gxp) * Lxp;
    const double Lb1 = pos_ref(gzm) * Lzm, Lb2 = neg_ref(gzp) * Lzp;
    if (fabs((a1 - a2) / dx + (b1 - b2) / dz) > 1e-9)
        return ((La1 - La2) / dx + (Lb1 - Lb2) / dz) / ((a1 - a2) / dx + (b1 - b2) / dz);
    return 0.0;
}

// Fast adjoint forms (see kernels3d.cu): den = sum_m w_m max(-e_m, 0),
// num = sum_m w_m max(e_m, 0) lambda_m with e_m = T_m - T0.
template <typename R>
__device__ __forceinline__ void adj2_terms(R T0, R Txp, R Txm, R Tzp, R Tzm, R Lxp, R Lxm, R Lzp, R Lzm, R wx, R wz,
                                           R& num, R& den) {
    const R z = R(0);
    R e;
    e = Txp - T0; den = wx * fmax(-e, z); num = wx * fmax(e, z) * Lxp;
    e = Txm - T0; den = fma(wx, fmax(-e, z), den); num = fma(wx * fmax(e, z), Lxm, num);
    e = Tzp - T0; den = fma(wz, fmax(-e, z), den); num = fma(wz * fmax(e, z), Lzp, num);
    e = Tzm - T0; den = fma(wz, fmax(-e, z), den); num = fma(wz * fmax(e, z), Lzm, num);
}

__device__ __forceinline__ float adj2_bulk(float T0, float Txp, float Txm, float Tzp, float Tzm, float Lxp, float Lxm,
                                           float Lzp, float Lzm, float wx, float wz) {
    const float ti = INFINITY;
    if (Txp >= ti || T0 >= ti || Txm >= ti || Tzp >= ti || Tzm >= ti) return 0.f;
    float num, den;
    adj2_terms<float>(T0, Txp, Txm, Tzp, Tzm, Lxp, Lxm, Lzp, Lzm, wx, wz, num, den);
    return (fabsf(den) > 1e-9f) ? __fdividef(num, den) : 0.f;
}

// FP64 polish adjoint update in residual-correction form (see kernels3d.cu): with mu_m =
// lambda_m where e_m > 0 and lambda0 where e_m < 0, r = num - den*lambda0 = sum_m w_m e_m mu_m
// in FP64 (11 FP64 instructions); den only scales the step and is FP32.  big: the FP32 step
// leaves a remainder above the floor.
__device__ __forceinline__ double adj2_polish(double T0, double Txp, double Txm, double Tzp, double Tzm, double Lxp,
                                              double Lxm, double Lzp, double Lzm, double L0, double wx, double wz,
                                              float wxf, float wzf, float floor, bool& big, float& dstep) {
    dstep = INFINITY;   // the branches that reset lambda to 0
    const long long inf = dbits(kInf);   // T >= INF on the bit patterns (T >= 0)
    if (dbits(Txp) >= inf || dbits(T0) >= inf || dbits(Txm) >= inf || dbits(Tzp) >= inf || dbits(Tzm) >= inf)
        return 0.0;
    const double exp_ = Txp - T0, exm = Txm - T0, ezp = Tzp - T0, ezm = Tzm - T0;
    auto mu = [&](double e, double L) { return __double2hiint(e) < 0 ? L0 : L; };
    auto nf = [](double e) { return __double2hiint(e) < 0 ? -narrow_trunc(e) : 0.0f; };   // max(-e, 0)
    const double r = fma(wx, fma(exp_, mu(exp_, Lxp), exm * mu(exm, Lxm)),
                         wz * fma(ezp, mu(ezp, Lzp), ezm * mu(ezm, Lzm)));
    const float den = wxf * (nf(exp_) + nf(exm)) + wzf * (nf(ezp) + nf(ezm));
    if (!(den > 1e-9f)) return 0.0;
    const float step = __fdividef(narrow_trunc(r), den);
    const float tol = floor * (1.0f + fabsf(narrow_trunc(L0)));
    big = fabsf(step) * 1.2e-7f > tol;
    dstep = fabsf(step);
    // corrections far below the convergence tolerance are dropped (bitwise fixed point, tiles lock)
    return fabsf(step) <= tol ? L0 : L0 + widen_exact(step);
}

// FP64 polish Godunov update, one Newton step on f(q) = wx max(q-a,0)^2 + wz max(q-b,0)^2 - s^2
// (FP64 differences and residual, 8 FP64 instructions; FP32 derivative and step); a: x-neighbour
// minimum, b: z-neighbour minimum.  big: the step's second-order remainder exceeds the floor.
__device__ __forceinline__ double eik2_newton(double U0, double a, double b, double s, double dx, double dz, double wx,
                                              double wz, float wxf, float wzf, float floor, bool& big,
                                              float& dstep) {
    const double px = pos_sign(U0 - a), pz = pos_sign(U0 - b);
    const double f = fma(wx * px, px, fma(wz * pz, pz, -s * s));
    const float fp = 2.0f * (wxf * narrow_trunc(px) + wzf * narrow_trunc(pz));
    if (!(fp > 0.0f)) {
        big = true;
        dstep = INFINITY;   // a restart: the change is not a Newton step
        return fmin(fma(dx, s, a), fma(dz, s, b));
    }
    const float step = __fdividef(narrow_trunc(f), fp);
    const float sw = (dbits(px) > 0 ? wxf : 0.0f) + (dbits(pz) > 0 ? wzf : 0.0f);
    big = sw * step * step > floor * fp;
    dstep = fabsf(step);   // the change of the node, to FP32 precision
    return fabsf(step) <= floor ? U0 : U0 - widen_exact(step);   // bitwise fixed point once converged
}

// Ordered integer of a value >= 0 (its bit pattern), FP32 or FP64.
__device__ __forceinline__ long long obits2(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ long long obits2(float x) { return __float_as_int(x); }

// Bitwise equality of two field values (FP32 or FP64).
template <typename Real>
__device__ __forceinline__ bool bits_same(Real a, Real b) {
    if constexpr (sizeof(Real) == 8) return __double_as_longlong(a) == __double_as_longlong(b);
    else return __float_as_uint(a) == __float_as_uint(b);
}

// ----------------------------------------------------------- quadrant selection (2D polish)
// Sweep order o: bit 0 = columns ascending, bit 1 = rows ascending.  The 2D form of the 3D
// octant selection: a polish update runs only in the orders that visit the node's active
// upwind neighbours (forward) / its larger-traveltime neighbours (adjoint) first.
constexpr unsigned kAscX2 = 0xa, kDescX2 = 0x5, kAscZ2 = 0xc, kDescZ2 = 0x3;

__device__ __forceinline__ unsigned fwd_orders2(long long u, long long xlo, long long xhi, long long zlo,
                                                long long zhi) {
    unsigned m = 0xf;
    if (u > (xlo < xhi ? xlo : xhi)) m &= xlo < xhi ? kAscX2 : (xhi < xlo ? kDescX2 : 0xfu);
    if (u > (zlo < zhi ? zlo : zhi)) m &= zlo < zhi ? kAscZ2 : (zhi < zlo ? kDescZ2 : 0xfu);
    return m;
}

__device__ __forceinline__ unsigned adj_orders2(long long t, long long xlo, long long xhi, long long zlo,
                                                long long zhi) {
    unsigned m = 0xf;
    const bool a = xlo > t, b = xhi > t, c = zlo > t, e = zhi > t;
    if (a != b) m &= a ? kAscX2 : kDescX2;
    if (c != e) m &= c ? kAscZ2 : kDescZ2;
    return m;
}

template <typename Dst, typename Src, typename Conv>
__device__ __forceinline__ void load_box2(Dst* box, const Src* __restrict__ g, int i0, int j0, int nr, int nc,
                                          Dst fill, int lane, Conv conv) {
    constexpr int NE = H2I * H2J;
    constexpr int BATCH = 16;
#pragma unroll 1
    for (int base = 0; base < NE; base += 32 * BATCH) {
        Dst v[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int e = base + u * 32 + lane;
            v[u] = fill;
            if (e < NE) {
                const int y = e / H2J, x = e - y * H2J;
                const int gi = i0 - 1 + y, gj = j0 - 1 + x;
                if ((unsigned)gi < (unsigned)nr && (unsigned)gj < (unsigned)nc) v[u] = conv(g[(long long)gi * nc + gj]);
            }
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int e = base + u * 32 + lane;
            if (e < NE) {
                const int y = e / H2J, x = e - y * H2J;
                box[y * R2 + x] = v[u];
            }
        }
    }
}

struct Ident2 {
    template <typename T> __device__ __forceinline__ T operator()(T v) const { return v; }
};

// Initial lock words from the field a phase starts from (as in the 3D sweeps): a tile is due
// in every order only if its halo box holds a reached traveltime (forward) or a nonzero lambda
// (adjoint); otherwise it is a fixed point of the update until a neighbour's change marks it.
// SEL (the adjoint polish): an idle tile keeps all four orders selected (bits 4-7), so that a
// neighbour's mark makes it due, and a tile counts as live only where some |lambda| exceeds a
// quarter of the polish floor (smaller values give corrections within the floor).  One warp per tile, lane = column of the box rows.
template <typename Real, bool ADJ, bool SEL>
__global__ void seed_tiles2_kernel(const Sweep2Args A) {
    const double thr = 0.25 * (double)A.polish_floor;   // SEL (adjoint polish): |lambda| above it
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= A.ntiles) return;   // whole warps
    const int q = A.act[blockIdx.y];
    const int lane = threadIdx.x & 31;
    const int nr = A.nr, nc = A.nc;
    const Real* f = reinterpret_cast<const Real*>(A.field) + A.inst_off[q];
    const int i0 = (t / A.nbj) * T2I, j0 = (t % A.nbj) * T2J;
    bool live = false;
#pragma unroll 1
    for (int i = i0 - 1; i <= i0 + T2I && !live; ++i) {
        if ((unsigned)i >= (unsigned)nr) continue;
        bool v = false;
        for (int j = j0 - 1 + lane; j <= j0 + T2J; j += 32) {
            if ((unsigned)j >= (unsigned)nc) continue;
            const Real x = __ldg(f + (long long)i * nc + j);
            if constexpr (ADJ && SEL) v |= dbits(fabs(x)) > dbits(thr);
            else v |= ADJ ? (x != Real(0)) : (x < Real(kInf));
        }
        live = __any_sync(0xffffffffu, v);
    }
    if (lane == 0) A.dirty[(long long)q * A.ntiles + t] = live ? 0xff : (SEL ? 0xf0 : 0);
}

template <int KIND>
__global__ void __launch_bounds__(kWarps2 * 32) sweep2d_kernel(const Sweep2Args A, const int d) {
    using Real = typename Traits2<KIND>::Real;
    using Aux = typename Traits2<KIND>::Aux;
    constexpr bool ADJ = Traits2<KIND>::adj;
    extern __shared__ __align__(16) unsigned char smem_raw[];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int d0 = A.diag_off[d];
    const int tile_idx = blockIdx.x * kWarps2 + warp;
    if (tile_idx >= A.diag_off[d + 1] - d0) return;
    int iter = A.iter;
    if (A.dyn) {   // replayed iteration graph
        if ((int)blockIdx.y >= __ldcg(A.dyn + 1)) return;
        iter = __ldcg(A.dyn);
    }
    const int q = A.act[blockIdx.y];

    const unsigned pk = A.diag_tiles[d0 + tile_idx];
    const bool py = A.dir & 2, px = A.dir & 1;
    const int bif = pk & 0xffff, bjf = pk >> 16;
    const int ti = py ? bif : A.nbi - 1 - bif;
    const int tj = px ? bjf : A.nbj - 1 - bjf;
    // tile locking, as in the 3D sweeps: bits 0-3 = orders still to process, bits 4-7 (polish)
    // = orders in which some node of the tile is selected
    constexpr bool kSelective = (KIND == kFwdPolish64 || KIND == kAdjPolish64);
    const int tid = ti * A.nbj + tj;
    int* dirty = A.dirty + (long long)q * A.ntiles;
    const int dm = __ldcg(dirty + tid);
    const int obit = 1 << A.dir;
    const int omask = kSelective ? (dm >> 4) & 0xf : 0xf;
    if (!(dm & omask & obit)) return;   // locked for this order (warp-uniform)
    __syncwarp();
    // Convergence test of the mixed kinds (FP32 bulk, polish): a node that moved by more than
    // the tolerance in some processing of this outer iteration, ORed over the iteration (a
    // polish change is its FP32 step).  The plain kinds compare with a snapshot taken at the
    // tile's first processing in the iteration, as the reference's isconv does.
    constexpr bool kSnap = KIND == kFwdPlain64 || KIND == kAdjPlain64;
    // the tile's lock word as lane 0 last wrote it (no other tile of this launch writes it)
    int dword = kSelective ? (dm & ~obit) : 0;
    if (lane == 0) {
        dirty[tid] = dword;
        if (A.work) atomicAdd(A.work + q, (unsigned long long)(min(T2I, A.nr - ti * T2I) * min(T2J, A.nc - tj * T2J)));
    }
    const int i0 = ti * T2I, j0 = tj * T2J;
    const int nr = A.nr, nc = A.nc;
    const int ei = min(T2I, nr - i0), ej = min(T2J, nc - j0);
    const long long n = (long long)nr * nc;

    Real* box = reinterpret_cast<Real*>(smem_raw + warp * warp_smem2<KIND>());
    Aux* tbox = reinterpret_cast<Aux*>(reinterpret_cast<unsigned char*>(box) + H2I * R2 * sizeof(Real));
    Real* fld = reinterpret_cast<Real*>(A.field) + A.inst_off[q];
    Real* snp = kSnap ? reinterpret_cast<Real*>(A.snap) + q * n : nullptr;

    const Real fill = ADJ ? Real(0) : Real(INFINITY);
    load_box2(box, fld, i0, j0, nr, nc, fill, lane, Ident2());

    const int lif = lane;
    const bool lane_ok = lif < ei;
    const int li = py ? lif : ei - 1 - lif;
    const int gi = i0 + li;
    unsigned fixed_lo = 0, fixed_hi = 0;
    if constexpr (ADJ) {
        const double* T = reinterpret_cast<const double*>(A.aux) + A.aux_off[q];
        if constexpr (!t_windows2<KIND>()) {
            // offsets from the tile corner's traveltime, formed without FP64 instructions
            const long long inf = dbits(kInf);
            double tr = T[(long long)i0 * nc + j0];
            if (dbits(tr) >= inf) tr = 0.0;
            load_box2(tbox, T, i0, j0, nr, nc, Aux(0), lane,
                      [tr, inf](double v) { return dbits(v) >= inf ? (Aux)INFINITY : (Aux)offset_f32(v, tr); });
        }
        if (lane_ok) {
            const unsigned* mrow = A.mask + A.mask_off[q] + (long long)gi * A.wpr + (j0 >> 5);
            fixed_lo = mrow[0];
            if ((j0 >> 5) + 1 < A.wpr) fixed_hi = mrow[1];
        }
    }

    // snapshot at the tile's first processing in this outer iteration (plain kinds)
    if constexpr (kSnap) {
        int* stamp = A.stamp + (long long)q * A.ntiles;
        if (__ldcg(stamp + tid) != iter) {
            for (int y = 0; y < ei; ++y)
                for (int x = lane; x < ej; x += 32) snp[(long long)(i0 + y) * nc + j0 + x] = box[(y + 1) * R2 + x + 1];
            if (lane == 0) stamp[tid] = iter;
        }
    }
    __syncwarp();
    bool moved = false;
    const float tabs_f = narrow_trunc(A.tol_abs), trel_f = narrow_trunc(A.tol_rel);   // FP32 kinds' test
    // the mixed kinds' test at a changed node (old -> nv; dstep: the polish step's size)
    auto note_move = [&](Real old, Real nv, float dstep) {
        if constexpr (kSelective) {
            if (dstep > tabs_f) moved = true;
        } else if constexpr (!kSnap) {
            if (fabsf(old - nv) > tabs_f + trel_f * fabsf(nv)) moved = true;
        }
    };

    int lim_row = -1, si = -1, sj = -1;
    if (A.inst_lim[q] >= 0) lim_row = A.inst_lim[q];
    if (A.inst_src[q] >= 0) { si = A.inst_src[q] >> 16; sj = A.inst_src[q] & 0xffff; }
    const int* rl = lim_row >= 0 ? A.rowlim + (long long)lim_row * nc : nullptr;
    const Aux* slow = reinterpret_cast<const Aux*>(A.aux);
    const bool row_interior = gi >= 1 && gi <= nr - 2;

    const float wx = A.wxf, wz = A.wzf, rsum = A.rsumf;
    const int cb = (li + 1) * R2 + 1;
    const int steps = ei + ej - 1;
    bool chg = false, chg_jlo = false, chg_jhi = false;
    unsigned sel = 0;
    // Face marks and own re-marking as in the 3D sweeps: only where the neighbour's node depends on
    // the changed one (forward: a neighbour below the node's value; adjoint: a larger traveltime;
    // with the margins of the plain kinds there).
    bool m_ilo = false, m_ihi = false;
    bool restep = false;   // polish: a remainder above the floor (visit again in this order)
    bool stale = false;    // plain, FP32 bulk: a changed node feeds an in-tile node visited before it

    // ---- adjoint traveltime of the FP64 kinds through register windows (as in the 3D sweeps):
    // lane lif (flipped row) is at flipped column jf = t - lif in step t and keeps its row's
    // traveltimes at jf-1, jf, jf+1 (loads issued three steps ahead); lane lif-1 is one column
    // ahead and lane lif+1 one behind, so their windows hold the rows above and below at jf;
    // lanes 0 and ei-1 read the halo rows outside the tile at their own position.
    constexpr bool TWIN2 = t_windows2<KIND>();
    const double* Tq = TWIN2 ? reinterpret_cast<const double*>(A.aux) + A.aux_off[q] : nullptr;
    const int glo = i0 + (py ? -1 : ei), ghi = i0 + (py ? ei : -1);   // rows of flipped rows -1 and ei
    const double* trow = (TWIN2 && lane_ok) ? Tq + (long long)gi * nc : nullptr;
    const double* hlrow = (TWIN2 && lif == 0 && (unsigned)glo < (unsigned)nr) ? Tq + (long long)glo * nc : nullptr;
    const double* hhrow =
        (TWIN2 && lif == ei - 1 && (unsigned)ghi < (unsigned)nr) ? Tq + (long long)ghi * nc : nullptr;
    auto tl = [&](const double* r, int p, int plo, int phi) -> double {
        const int g = j0 + (px ? p : ej - 1 - p);
        return (r != nullptr && p >= plo && p <= phi && (unsigned)g < (unsigned)nc) ? __ldg(r + g) : 0.0;
    };
    double tm = 0.0, t0w = 0.0, tp = 0.0, q1 = 0.0, q2 = 0.0;
    double hl0 = 0.0, hl1 = 0.0, hl2 = 0.0, hh0 = 0.0, hh1 = 0.0, hh2 = 0.0;
    if constexpr (TWIN2) {
        const int f0 = -lif;
        tm = tl(trow, f0 - 1, -1, ej); t0w = tl(trow, f0, -1, ej); tp = tl(trow, f0 + 1, -1, ej);
        q1 = tl(trow, f0 + 2, -1, ej); q2 = tl(trow, f0 + 3, -1, ej);
        hl0 = tl(hlrow, f0, 0, ej - 1); hl1 = tl(hlrow, f0 + 1, 0, ej - 1); hl2 = tl(hlrow, f0 + 2, 0, ej - 1);
        hh0 = tl(hhrow, f0, 0, ej - 1); hh1 = tl(hhrow, f0 + 1, 0, ej - 1); hh2 = tl(hhrow, f0 + 2, 0, ej - 1);
    }

#pragma unroll 1
    for (int t = 0; t < steps; ++t) {
        const int ljf = t - lif;
        // adjoint: the traveltimes around this lane's node, in grid orientation
        Aux T0 = Aux(0), Txm = Aux(0), Txp = Aux(0), Tzm = Aux(0), Tzp = Aux(0);
        if constexpr (TWIN2) {
            const double up = __shfl_sync(0xffffffffu, tm, (lane - 1) & 31);
            const double dn = __shfl_sync(0xffffffffu, tp, (lane + 1) & 31);
            const double fim = lif == 0 ? hl0 : up, fip = lif == ei - 1 ? hh0 : dn;
            T0 = t0w;
            Txm = px ? tm : tp; Txp = px ? tp : tm;
            Tzm = py ? fim : fip; Tzp = py ? fip : fim;
        }
        if (lane_ok && ljf >= 0 && ljf < ej) {
            const int lj = px ? ljf : ej - 1 - ljf;
            const int c = cb + lj;
            const int gj = j0 + lj;
            if constexpr (!ADJ) {
                // the source node (and the opt-in fixed region around it) keeps its value
                const bool upd = (rl == nullptr || gi <= __ldg(rl + gj)) &&
                                 (si < 0 || (gi - si) * (gi - si) + (gj - sj) * (gj - sj) > A.src_r2);
                if (upd) {
                    const Real old = box[c];
                    Real nv = old;
                    float dstep = INFINITY;   // polish: the size of this node's change
                    const Real bz = ref_min(box[c - R2], box[c + R2]);
                    const Real ax = ref_min(box[c + 1], box[c - 1]);
                    const Real s = __ldg(slow + (long long)gi * nc + gj);
                    if constexpr (KIND == kFwdPlain64) {
                        const double qv = eik2_plain(ax, bz, s, A);
                        nv = ref_min(old, qv);
                    } else if constexpr (KIND == kFwdFast32) {
                        const float qv = eik2_fast<float>(ax, bz, s, A.dxf, A.dzf, wx, wz, rsum);
                        nv = ref_min(old, qv);
                    } else {
                        const unsigned m = fwd_orders2(dbits(old), dbits(box[c - 1]), dbits(box[c + 1]),
                                                       dbits(box[c - R2]), dbits(box[c + R2]));
                        sel |= m;
                        if (m & obit) {
                            bool big = false;
                            nv = eik2_newton(old, ax, bz, s, A.dx, A.dz, A.inv2x, A.inv2z, A.wxf, A.wzf,
                                             A.polish_floor, big, dstep);
                            restep |= big;
                        }
                    }
                    if (!bits_same(old, nv)) {
                        box[c] = nv;
                        chg = true;
                        note_move(old, nv, dstep);
                        // (plain: as forward_depends_exact without a limit, since a discriminant that rounds
                        // below 0 gives the unreached value here, and no third neighbour comes in)
                        auto dep = [&](int n) {
                            constexpr long long kMargin = KIND == kFwdPlain64 ? 1ll << 33 : 0;
                            return min(obits2(old), obits2(nv)) < obits2(box[n]) + kMargin;
                        };
                        if (li == 0 && dep(c - R2)) m_ilo = true;
                        if (li == ei - 1 && dep(c + R2)) m_ihi = true;
                        if (lj == 0 && dep(c - 1)) chg_jlo = true;
                        if (lj == ej - 1 && dep(c + 1)) chg_jhi = true;
                        if constexpr (!kSelective) {
                            if (lif > 0 && dep(py ? c - R2 : c + R2)) stale = true;
                            if (ljf > 0 && dep(px ? c - 1 : c + 1)) stale = true;
                        }
                    }
                }
            } else {
                const unsigned fb = lj < 32 ? (fixed_lo >> lj) : (fixed_hi >> (lj - 32));
                if (row_interior && gj >= 1 && gj <= nc - 2 && !(fb & 1u)) {
                    const Real old = box[c];
                    Real r = old;
                    float dstep = INFINITY;   // polish: the size of this node's change
                    if constexpr (!TWIN2) {   // FP32 bulk: from the staged offsets
                        T0 = tbox[c]; Txp = tbox[c + 1]; Txm = tbox[c - 1]; Tzp = tbox[c + R2]; Tzm = tbox[c - R2];
                    }
                    if constexpr (KIND == kAdjPlain64) {
                        r = adj2_plain(T0, Txp, Txm, Tzp, Tzm, box[c + 1], box[c - 1], box[c + R2], box[c - R2], A);
                    } else if constexpr (KIND == kAdjFast32) {
                        r = adj2_bulk(T0, Txp, Txm, Tzp, Tzm, box[c + 1], box[c - 1], box[c + R2], box[c - R2], wx, wz);
                    } else {
                        const unsigned m = adj_orders2(dbits(T0), dbits(Txm), dbits(Txp), dbits(Tzm), dbits(Tzp));
                        sel |= m;
                        if (m & obit) {
                            bool big = false;
                            r = adj2_polish(T0, Txp, Txm, Tzp, Tzm, box[c + 1], box[c - 1], box[c + R2], box[c - R2],
                                            old, A.inv2x, A.inv2z, A.wxf, A.wzf, A.polish_floor, big, dstep);
                            restep |= big;
                        }
                    }
                    if (!bits_same(old, r)) {
                        box[c] = r;
                        chg = true;
                        note_move(old, r, dstep);
                        // lambda at the neighbour node reads this node if its traveltime is larger
                        // (FP32 bulk: offsets from the tile's corner, compared as values)
                        auto dep = [&](Aux tn, int n) {
                            if constexpr (KIND == kAdjPlain64)
                                return adj_depends_exact(T0, tn, box[n], old, r);
                            else if constexpr (sizeof(Aux) == 8) return obits2(T0) > obits2(tn);
                            else return T0 > tn;
                        };
                        if (li == 0 && dep(Tzm, c - R2)) m_ilo = true;
                        if (li == ei - 1 && dep(Tzp, c + R2)) m_ihi = true;
                        if (lj == 0 && dep(Txm, c - 1)) chg_jlo = true;
                        if (lj == ej - 1 && dep(Txp, c + 1)) chg_jhi = true;
                        if constexpr (!kSelective) {
                            if (lif > 0 && dep(py ? Tzm : Tzp, py ? c - R2 : c + R2)) stale = true;
                            if (ljf > 0 && dep(px ? Txm : Txp, px ? c - 1 : c + 1)) stale = true;
                        }
                    }
                }
            }
        }
        if constexpr (TWIN2) {   // slide the windows to step t + 1
            tm = t0w; t0w = tp; tp = q1; q1 = q2; q2 = tl(trow, t + 4 - lif, -1, ej);
            hl0 = hl1; hl1 = hl2; hl2 = tl(hlrow, t + 3 - lif, 0, ej - 1);
            hh0 = hh1; hh1 = hh2; hh2 = tl(hhrow, t + 3 - lif, 0, ej - 1);
        }
        __syncwarp();
    }

    if constexpr (kSelective) {
        const unsigned tsel = __reduce_or_sync(0xffffffffu, sel);
        dword = (dword & 0xf) | (int)(tsel << 4);
        if (lane == 0) dirty[tid] = dword;
    }
    // nothing changed: the field and its convergence flag stand as they are
    if (!__any_sync(0xffffffffu, chg)) return;
    // unlock this tile and the face neighbours that see a changed face node (lane = row)
    const unsigned f_ilo = __ballot_sync(0xffffffffu, m_ilo);
    const unsigned f_ihi = __ballot_sync(0xffffffffu, m_ihi);
    const unsigned f_jlo = __ballot_sync(0xffffffffu, chg_jlo);
    const unsigned f_jhi = __ballot_sync(0xffffffffu, chg_jhi);
    // own re-marking (see the 3D sweeps): a polish tile stays locked in this order after
    // updates with remainders below the floor; a plain or FP32 bulk tile none of whose changed nodes
    // feeds an already visited node is a fixed point until a neighbour marks it
    bool again = true;
    if constexpr (kSelective) again = __any_sync(0xffffffffu, restep);
    else again = __any_sync(0xffffffffu, stale);
    if (lane == 0) {
        dirty[tid] = dword | (again ? 0xf : (kSelective ? (0xf & ~obit) : 0));
        if (f_ilo && ti > 0) atomicOr(dirty + tid - A.nbj, 0xf);
        if (f_ihi && ti < A.nbi - 1) atomicOr(dirty + tid + A.nbj, 0xf);
        if (f_jlo && tj > 0) atomicOr(dirty + tid - 1, 0xf);
        if (f_jhi && tj < A.nbj - 1) atomicOr(dirty + tid + 1, 0xf);
    }
    for (int y = 0; y < ei; ++y) {
        for (int x = lane; x < ej; x += 32) {
            const long long at = (long long)(i0 + y) * nc + j0 + x;
            const Real v = box[(y + 1) * R2 + x + 1];
            fld[at] = v;
            if constexpr (kSnap) {   // isconv (equal bits need no FP64 instruction)
                const Real was = __ldcg(snp + at);
                if (!bits_same(was, v) && fabs(was - v) > A.tol_abs + A.tol_rel * fabs(v)) moved = true;
            }
        }
    }
    const bool any_moved = __any_sync(0xffffffffu, moved);
    if constexpr (kSnap) {
        if (lane == 0) A.diff[(long long)q * A.ntiles + tid] = any_moved ? 1 : 0;
    } else {
        if (lane == 0 && any_moved) A.diff[(long long)q * A.ntiles + tid] = 1;
    }
}

// ----------------------------------------------------------- strips schedule
// One launch per phase: a block solves an instance, one warp per strip of T2I rows (lane = row).  A
// warp streams along its strip, one column per step, lane lif one column behind lane lif - 1, and
// the warp of the strip downstream follows it some columns behind, so that a sweep takes about
// ncols + nrows steps instead of the 95 per tile of a launch per tile diagonal, without its
// launches, box loads and ramps (601 x 201 nodes: 2900 steps an iteration against 6100).  A sweep
// order begins on a strip as soon as the strip that is downstream of it has left the columns.
//
// What is processed, and with what values, is exactly what the per-diagonal launches process: the
// strip is cut into the same T2I x T2J tiles with the same lock words, and a tile is visited in an
// order only when it is due in it at the time its turn comes there.  A tile already due when the
// warp reaches it starts at once, while its upstream strip and the tile before it are still
// unfinished; otherwise the warp waits for both (they may mark it) and then visits or skips it.
//   lock words  a visit takes its order's bit (plain, FP32 bulk: all order bits) atomically when it
//               starts and writes the word when it ends, after the upstream strip's tile has
//               ended, so that marks that come from tiles before it in the same order are dropped
//               (plain, FP32 bulk) or kept for the other orders (polish), as if they had come first;
//   tdone       per tile: sweep orders of this iteration that are complete, marks included;
//   prog        per strip: order * (nc + 1) + columns whose values are final in that order.
// Field values: a lane keeps its row's new value at jf - 1 and old values at jf .. jf + 3 in
// registers (loads issued three steps ahead, a cache line serves 16 or 32 steps), neighbour rows
// come by warp shuffle, and the rows that face a neighbouring strip are kept in shared memory.
// All waits are on warps of the same block and are bounded (two seconds, then *err).
constexpr int kStripMax = 16;       // strips (warps) of a block
constexpr int kProgStep = 8;        // columns between two progress reports

template <int KIND>
inline size_t strips_smem(int nr, int nc) {
    const size_t ns = (nr + T2I - 1) / T2I, nbj = (nc + T2J - 1) / T2J;
    const size_t faces = 2 * ns * nc * sizeof(typename Traits2<KIND>::Real);
    return (faces + 15) / 16 * 16 + sizeof(int) * (4 * ns * nbj + ns + nc);
}

__device__ __forceinline__ unsigned long long strip_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// A lane's view of its warp for strip_sync.h.
struct StripWarp {
    int lane;
    int* abort;
    __device__ __forceinline__ bool leader() const { return lane == 0; }
    __device__ __forceinline__ void barrier() const { __syncwarp(); }
    __device__ __forceinline__ void fence() const { __threadfence_block(); }
    __device__ __forceinline__ void store(volatile int* p, int v) const { *p = v; }
    __device__ __forceinline__ int broadcast(int v) const { return __shfl_sync(0xffffffffu, v, 0); }
    // until *p >= want (a word of another warp of this block), two seconds at most; 0: given up
    __device__ __forceinline__ int poll(volatile int* p, int want) const {
        unsigned long long since = 0;
        for (int spin = 0; *p < want; ++spin) {
            if (*(volatile int*)abort) return 0;
            if (spin > 16) __nanosleep(40);
            if ((spin & 1023) == 1023) {
                const unsigned long long now = strip_ns();
                if (!since) since = now;
                else if (now - since > 2000000000ull) { *(volatile int*)abort = 1; return 0; }
            }
        }
        return 1;
    }
};

// Traveltimes for the FP32 bulk adjoint, per instance: split parts, +inf where unreached.  An offset
// from a tile's corner is then three FP32 operations per value; split in the step instead, the
// sweep took 12.5 ms for 40 + 40 instances of 601 x 201 nodes.
__global__ void split_inst_kernel(const double* __restrict__ a, float2* __restrict__ b, const long long* __restrict__ oa,
                                  const long long* __restrict__ ob, long long n) {
    const int q = blockIdx.y;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const double v = a[oa[q] + t];
        b[ob[q] + t] = dbits(v) >= dbits(kInf) ? make_float2(INFINITY, 0.0f) : split_hl(v);
    }
}
__device__ __forceinline__ double shfl_any(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float shfl_any(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float2 shfl_any(float2 v, int src) {
    return make_float2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

template <int KIND>
__global__ void __launch_bounds__(kStripMax * 32) sweep2d_strips(const Sweep2Args A, const int nact,
                                                                 const int* __restrict__ caps, int* __restrict__ queue,
                                                                 int* __restrict__ result) {
    using Real = typename Traits2<KIND>::Real;
    using Aux = typename Traits2<KIND>::Aux;
    constexpr bool ADJ = Traits2<KIND>::adj;
    constexpr bool OFFS = KIND == kAdjFast32;   // traveltimes as FP32 offsets from the tile's corner
    using TV = typename std::conditional<OFFS, float2, double>::type;
    constexpr bool kSelective = (KIND == kFwdPolish64 || KIND == kAdjPolish64);
    constexpr bool kSnap = KIND == kFwdPlain64 || KIND == kAdjPlain64;
    constexpr unsigned kChg = 1, kMoved = 2, kAgain = 4, kUp = 8, kDn = 16, kPrev = 32, kNext = 64;   // + selected orders << 8
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_item, s_abort;
    const int nr = A.nr, nc = A.nc, ns = A.nbi, nbj = A.nbj, ntiles = A.ntiles;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nthr = blockDim.x;
    Real* face = reinterpret_cast<Real*>(smem_raw);   // [2][ns][nc]: first and last row of every strip
    int* s_dirty = reinterpret_cast<int*>(smem_raw + (2 * sizeof(Real) * ns * nc + 15) / 16 * 16);
    int* s_diff = s_dirty + ntiles;
    int* s_stamp = s_diff + ntiles;
    volatile int* s_tdone = s_stamp + ntiles;
    volatile int* s_prog = s_tdone + ntiles;
    int* s_rl = s_stamp + 2 * ntiles + ns;
    const int i0 = w * T2I, ei = min(T2I, nr - i0), last = ei - 1;
    const Real fill = ADJ ? Real(0) : Real(INFINITY);
    const float tabs_f = narrow_trunc(A.tol_abs), trel_f = narrow_trunc(A.tol_rel);
    const StripWarp warp{lane, &s_abort};
    auto wait_for = [&](volatile int* p, int want) -> bool { return strip_wait(warp, p, want); };   // warp-uniform
    auto tile_end = [&](int cf, bool px) { return min(nc, px ? (cf + 1) * T2J : nc - (nbj - 1) * T2J + cf * T2J); };

    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(queue, 1);
        __syncthreads();
        const int item = s_item;
        __syncthreads();
        if (item >= nact) return;   // block-uniform
        const int q = A.act[item], cap = caps[item];
        Real* fld = reinterpret_cast<Real*>(A.field) + A.inst_off[q];
        Real* snp = kSnap ? reinterpret_cast<Real*>(A.snap) + (long long)q * nr * nc : nullptr;
        // adjoint: traveltime (FP32 bulk: split parts, +inf where unreached)
        const TV* Tq = ADJ ? reinterpret_cast<const TV*>(A.aux) + A.aux_off[q] : nullptr;
        const unsigned* mq = ADJ ? A.mask + A.mask_off[q] : nullptr;
        const bool lim = !ADJ && A.inst_lim[q] >= 0;
        int si = -1, sj = -1;
        if (!ADJ && A.inst_src[q] >= 0) { si = A.inst_src[q] >> 16; sj = A.inst_src[q] & 0xffff; }
        for (int t = threadIdx.x; t < ntiles; t += nthr) {
            s_dirty[t] = A.dirty[(long long)q * ntiles + t];
            s_stamp[t] = -1;
        }
        for (int e = threadIdx.x; e < ns * nc; e += nthr) {
            const int s = e / nc, j = e - s * nc;
            face[e] = fld[(long long)s * T2I * nc + j];
            face[ns * nc + e] = fld[(long long)min(s * T2I + T2I - 1, nr - 1) * nc + j];
        }
        if (lim)
            for (int j = threadIdx.x; j < nc; j += nthr) s_rl[j] = A.rowlim[(long long)A.inst_lim[q] * nc + j];
        if (threadIdx.x == 0) s_abort = 0;
        int it = 0;
        bool moved_any = true;
        while (it < cap) {
            for (int t = threadIdx.x; t < ntiles; t += nthr) {
                s_diff[t] = 0;
                s_tdone[t] = 0;
            }
            for (int s = threadIdx.x; s < ns; s += nthr) s_prog[s] = 0;
            __syncthreads();
            for (int o = 0; o < 4; ++o) {
                if (__any_sync(0xffffffffu, *(volatile int*)&s_abort)) break;   // warp-uniform
                const bool py = o & 2, px = o & 1;
                const int obit = 1 << o, pbase = o * (nc + 1);
                const int lif = lane;
                const bool lane_ok = lif < ei;
                const int li = py ? lif : last - lif, gi = i0 + li;
                const int us = py ? w - 1 : w + 1, ds = py ? w + 1 : w - 1;
                const bool hasU = (unsigned)us < (unsigned)ns, hasD = (unsigned)ds < (unsigned)ns;
                const Real* faceU = face + ((py ? ns : 0) + (hasU ? us : 0)) * nc;
                const Real* faceD = face + ((py ? 0 : ns) + (hasD ? ds : 0)) * nc;
                Real* ownTop = li == 0 ? face + w * nc : nullptr;
                Real* ownBot = li == last ? face + (ns + w) * nc : nullptr;
                Real* urow = fld + (long long)(lane_ok ? gi : i0) * nc;   // written where `on`
                const long long rowbase = (long long)(lane_ok ? gi : i0) * nc;
                auto gcol = [&](int p) { return px ? p : nc - 1 - p; };
                auto due = [&](int dm) { return (dm & (kSelective ? (dm >> 4) & 0xf : 0xf) & obit) != 0; };
                auto tile_at = [&](int cf) { return w * nbj + (px ? cf : nbj - 1 - cf); };
                auto strip_tile = [&](int s, int cf) { return s * nbj + (px ? cf : nbj - 1 - cf); };
                auto word = [&](int t) { return __shfl_sync(0xffffffffu, *(volatile int*)(s_dirty + t), 0); };
                bool ok = true;
                int cf = 0;
                while (cf < nbj && ok) {
                    // the strip downstream has this tile's values of the previous order
                    if (o > 0 && hasD) ok = wait_for(s_tdone + strip_tile(ds, cf), o);
                    if (!ok) break;
                    if (!due(word(tile_at(cf)))) {
                        if (hasU) ok = wait_for(s_tdone + strip_tile(us, cf), o + 1);
                        if (!ok) break;
                        if (!due(word(tile_at(cf)))) {   // locked in this order
                            strip_publish(warp, s_prog + w, pbase + tile_end(cf, px));
                            strip_publish(warp, s_tdone + tile_at(cf), o + 1);
                            ++cf;
                            continue;
                        }
                    }
                    // ---- stream from this tile on, over the tiles that are due when reached
                    const int js = cf ? tile_end(cf - 1, px) : 0;
                    int cA = cf, endA = tile_end(cf, px);   // the next tile to end
                    int cB = cf, endB = endA;               // the last tile begun (cA or cA + 1)
                    int startB = js;
                    bool firstA = false, firstB = false;    // plain: a tile's first visit of the iteration
                    float2 cornA = make_float2(0.f, 0.f), cornB = cornA;
                    auto begin = [&](int c, bool& first, float2& corn) {
                        const int t = tile_at(c);
                        int was = 0;
                        if (lane == 0) {
                            atomicAnd(s_dirty + t, kSelective ? ~obit : ~0xf);
                            if (A.work) atomicAdd(A.work + q, (unsigned long long)(ei * (tile_end(c, px) - (c ? tile_end(c - 1, px) : 0))));
                            if constexpr (kSnap) {
                                was = s_stamp[t] != it;
                                s_stamp[t] = it;
                            }
                        }
                        if constexpr (kSnap) first = __shfl_sync(0xffffffffu, was, 0);
                        if constexpr (OFFS) {   // an unreached corner counts as 0
                            corn = Tq[(long long)i0 * nc + (px ? c : nbj - 1 - c) * T2J];
                            if (corn.x == INFINITY) corn = make_float2(0.0f, 0.0f);
                        }
                    };
                    begin(cA, firstA, cornA);
                    firstB = firstA;
                    cornB = cornA;
                    int lstart = js, lend = endA;   // this lane's tile (flipped columns)
                    bool lfirst = firstA;
                    float2 lcorn = cornA;
                    unsigned cur = 0, prev = 0;     // what this lane found in its tile / in the one before
                    // Row values at flipped column p (clamped into the row: the update selects the fill
                    // at the ends); no branch, a lane without a row reads the strip's first.
                    auto clampc = [&](int p) { return gcol(min(max(p, 0), nc - 1)); };
                    const int f0 = js - lif;
                    Real um = urow[clampc(f0 - 1)], u0 = urow[clampc(f0)], up = urow[clampc(f0 + 1)];
                    Real uq1 = urow[clampc(f0 + 2)], uq2 = urow[clampc(f0 + 3)];
                    const Aux* srow = reinterpret_cast<const Aux*>(A.aux) + rowbase;   // forward: slowness
                    Aux s0 = Aux(0), s1 = Aux(0), s2 = Aux(0), s3 = Aux(0);
                    if constexpr (!ADJ) {
                        s0 = __ldg(srow + clampc(f0)); s1 = __ldg(srow + clampc(f0 + 1));
                        s2 = __ldg(srow + clampc(f0 + 2)); s3 = __ldg(srow + clampc(f0 + 3));
                    }
                    Real n0 = Real(0), n1 = Real(0);   // plain: the snapshot at jf, jf + 1
                    if constexpr (kSnap) { n0 = snp[rowbase + clampc(f0)]; n1 = snp[rowbase + clampc(f0 + 1)]; }
                    // adjoint: traveltimes of the row at jf-1 .. jf+3, and of the rows next to the strip
                    const TV* trow = Tq + rowbase;
                    const int gu = i0 + (py ? -1 : ei), gd = i0 + (py ? ei : -1);
                    const bool ownU = ADJ && lif == 0 && (unsigned)gu < (unsigned)nr;
                    const bool ownD = ADJ && lif == last && (unsigned)gd < (unsigned)nr;
                    const TV* hurow = Tq + (long long)(ownU ? gu : i0) * nc;
                    const TV* hdrow = Tq + (long long)(ownD ? gd : i0) * nc;
                    auto hload = [&](bool own, const TV* r, int p) -> TV {
                        TV v{};
                        if (own) v = __ldg(r + clampc(p));
                        return v;
                    };
                    TV tm{}, t0{}, tp{}, tq1{}, tq2{}, hu0{}, hu1{}, hu2{}, hd0{}, hd1{}, hd2{};
                    unsigned fcur = 0, fnext = 0;   // fixed-node bits of the lane's 32-column block and of the next
                    int fblk = -1;
                    auto fload = [&](int blk) -> unsigned {
                        return lane_ok && blk >= 0 && blk < A.wpr ? mq[(long long)gi * A.wpr + blk] : 0u;
                    };
                    if constexpr (ADJ) {
                        tm = __ldg(trow + clampc(f0 - 1)); t0 = __ldg(trow + clampc(f0)); tp = __ldg(trow + clampc(f0 + 1));
                        tq1 = __ldg(trow + clampc(f0 + 2)); tq2 = __ldg(trow + clampc(f0 + 3));
                        hu0 = hload(ownU, hurow, f0); hu1 = hload(ownU, hurow, f0 + 1); hu2 = hload(ownU, hurow, f0 + 2);
                        hd0 = hload(ownD, hdrow, f0); hd1 = hload(ownD, hdrow, f0 + 1); hd2 = hload(ownD, hdrow, f0 + 2);
                        fblk = gcol(js) >> 5;
                        fcur = fload(fblk);
                        fnext = fload(fblk + (px ? 1 : -1));
                    }
                    const bool rowin = gi >= 1 && gi <= nr - 2;
                    const int qi2 = (gi - si) * (gi - si);
                    int ready = js;         // columns of the upstream strip known to be final
                    bool extend = true;
                    int t = 0;
                    for (;;) {
                        // ---- what has to be settled before lane 0's next column
                        const int jl = js + t;   // lane 0's column
                        if (jl == endB && extend) {   // lane 0 is through the last tile begun
                            extend = false;
                            // (a last tile narrower than the lanes' skew would end in some lanes before
                            // the tile ahead of it does in the others: it is begun afresh)
                            if (cB + 1 < nbj && tile_end(cB + 1, px) - endB >= T2I) {
                                if (o > 0 && hasD) ok = wait_for(s_tdone + strip_tile(ds, cB + 1), o);
                                if (!ok) break;
                                if (due(word(tile_at(cB + 1)))) {
                                    ++cB;
                                    startB = endB;
                                    endB = tile_end(cB, px);
                                    begin(cB, firstB, cornB);
                                    extend = true;
                                }
                            }
                        }
                        if (hasU && jl >= ready && jl < endB) {
                            ready = min(jl + kProgStep, endB);
                            ok = wait_for(s_prog + us, pbase + ready);
                            if (!ok) break;
                        }
                        // ---- steps up to the next such point, the end of tile cA or the next progress report
                        const int doneA = endA - js + last;   // steps after which every lane is through cA
                        int stop = min(t + kProgStep, doneA);
                        if (jl < endB) stop = min(stop, (hasU ? ready : endB) - js);
#pragma unroll 1
                        for (; t < stop; ++t) {
                            const int jf = js + t - lif, gj = clampc(jf);
                            const bool on = lane_ok & ((unsigned)(jf - js) < (unsigned)(endB - js));
                            // loads of the next steps first
                            const int g4 = clampc(jf + 4);
                            const Real uq3 = urow[g4];
                            Aux s4 = Aux(0);
                            if constexpr (!ADJ) s4 = __ldg(srow + g4);
                            Real n2 = Real(0);
                            if constexpr (kSnap) n2 = snp[rowbase + clampc(jf + 2)];
                            TV tq3{}, hu3{}, hd3{};
                            if constexpr (ADJ) {
                                tq3 = __ldg(trow + g4);
                                hu3 = hload(ownU, hurow, jf + 3);
                                hd3 = hload(ownD, hdrow, jf + 3);
                            }
                            // neighbour rows: upstream (new values) and downstream (old values)
                            Real U = shfl_any(um, (lane - 1) & 31), D = shfl_any(up, (lane + 1) & 31);
                            const Real fu = faceU[gj], fd = faceD[gj];
                            if (lif == 0) U = hasU ? fu : fill;
                            if (lif == last) D = hasD ? fd : fill;
                            const Real L = !ADJ && jf == 0 ? fill : um, R = !ADJ && jf == nc - 1 ? fill : up;
                            TV TU{}, TD{};
                            if constexpr (ADJ) {
                                TU = shfl_any(tm, (lane - 1) & 31);
                                TD = shfl_any(tp, (lane + 1) & 31);
                                if (lif == 0) TU = hu0;
                                if (lif == last) TD = hd0;
                            }
                            if constexpr (kSnap) lfirst = jf == lstart ? (lstart == startB ? firstB : firstA) : lfirst;
                            if constexpr (OFFS) {
                                if (jf == lstart) lcorn = lstart == startB ? cornB : cornA;
                            }
                            const Real old = u0;
                            Real nv = old;
                            float dstep = INFINITY;   // polish: the size of this node's change
                            bool upd = on;
                            // in grid orientation (p: index + 1, m: index - 1)
                            const Real Xp = px ? R : L, Xm = px ? L : R, Zp = py ? D : U, Zm = py ? U : D;
                            Aux oT0{}, oTxp{}, oTxm{}, oTzp{}, oTzm{};
                            if constexpr (!ADJ) {
                                if (lim) upd = upd & (gi <= s_rl[gj]);
                                if (si >= 0) upd = upd & (qi2 + (gj - sj) * (gj - sj) > A.src_r2);
                                const Real bz = ref_min(Zm, Zp), ax = ref_min(Xp, Xm);
                                if constexpr (KIND == kFwdPlain64) {
                                    if (upd) nv = ref_min(old, eik2_plain(ax, bz, s0, A));
                                } else if constexpr (KIND == kFwdFast32) {
                                    const float c = ref_min(old, eik2_fast_sel(ax, bz, s0, A.dxf, A.dzf, A.wxf, A.wzf, A.rsumf));
                                    nv = upd ? c : old;
                                } else {
                                    const unsigned m = fwd_orders2(dbits(old), dbits(Xm), dbits(Xp), dbits(Zm), dbits(Zp));
                                    cur |= upd ? m << 8 : 0u;
                                    if (upd & ((m & obit) != 0)) {
                                        bool big = false;
                                        nv = eik2_newton(old, ax, bz, s0, A.dx, A.dz, A.inv2x, A.inv2z, A.wxf, A.wzf,
                                                         A.polish_floor, big, dstep);
                                        cur |= big ? kAgain : 0u;
                                    }
                                }
                            } else {
                                const bool nblk = on & ((gj >> 5) != fblk);
                                if (nblk) {
                                    fblk = gj >> 5;
                                    fcur = fnext;
                                    fnext = fload(fblk + (px ? 1 : -1));
                                }
                                upd = on & rowin & ((unsigned)(gj - 1) < (unsigned)(nc - 2)) & !((fcur >> (gj & 31)) & 1u);
                                const TV vp_ = px ? tp : tm, vm_ = px ? tm : tp, wp_ = py ? TD : TU, wm_ = py ? TU : TD;
                                if constexpr (OFFS) {
                                    auto off = [&](float2 v) { return (v.x - lcorn.x) + (v.y - lcorn.y); };
                                    oT0 = off(t0); oTxp = off(vp_); oTxm = off(vm_); oTzp = off(wp_); oTzm = off(wm_);
                                } else {
                                    oT0 = t0; oTxp = vp_; oTxm = vm_; oTzp = wp_; oTzm = wm_;
                                }
                                if constexpr (KIND == kAdjPlain64) {
                                    if (upd) nv = adj2_plain(oT0, oTxp, oTxm, oTzp, oTzm, Xp, Xm, Zp, Zm, A);
                                } else if constexpr (KIND == kAdjFast32) {
                                    const float c = adj2_bulk(oT0, oTxp, oTxm, oTzp, oTzm, Xp, Xm, Zp, Zm, A.wxf, A.wzf);
                                    nv = upd ? c : old;
                                } else {
                                    const unsigned m = adj_orders2(dbits(oT0), dbits(oTxm), dbits(oTxp), dbits(oTzm), dbits(oTzp));
                                    cur |= upd ? m << 8 : 0u;
                                    if (upd & ((m & obit) != 0)) {
                                        bool big = false;
                                        nv = adj2_polish(oT0, oTxp, oTxm, oTzp, oTzm, Xp, Xm, Zp, Zm, old, A.inv2x,
                                                         A.inv2z, A.wxf, A.wzf, A.polish_floor, big, dstep);
                                        cur |= big ? kAgain : 0u;
                                    }
                                }
                            }
                            if constexpr (kSnap) {   // isconv against the value at the iteration's start
                                if (upd & lfirst) snp[rowbase + gj] = old;
                                const Real was = lfirst ? old : n0;
                                if (upd & !bits_same(was, nv))
                                    if (fabs(was - nv) > A.tol_abs) cur |= kMoved;
                            }
                            if (!bits_same(old, nv)) {
                                urow[gj] = nv;
                                if (ownTop) ownTop[gj] = nv;
                                if (ownBot) ownBot[gj] = nv;
                                cur |= kChg;
                                if constexpr (kSelective) {
                                    if (dstep > tabs_f) cur |= kMoved;
                                } else if constexpr (!kSnap) {
                                    if (fabsf(old - nv) > tabs_f + trel_f * fabsf(nv)) cur |= kMoved;
                                }
                                // does the neighbour (value vn, traveltime tn) depend on this node? (see the 3D sweeps)
                                auto dep = [&](Real vn, Aux tn) -> bool {
                                    if constexpr (!ADJ) {
                                        constexpr long long kMargin = KIND == kFwdPlain64 ? 1ll << 33 : 0;
                                        return min(obits2(old), obits2(nv)) < obits2(vn) + kMargin;
                                    } else if constexpr (KIND == kAdjPlain64) {
                                        return adj_depends_exact(oT0, tn, vn, old, nv);
                                    } else if constexpr (sizeof(Aux) == 8) {
                                        return obits2(oT0) > obits2(tn);
                                    } else {
                                        return oT0 > tn;
                                    }
                                };
                                const Aux au = py ? oTzm : oTzp, ad = py ? oTzp : oTzm, al = px ? oTxm : oTxp, ar = px ? oTxp : oTxm;
                                const bool du = dep(U, au), dl = dep(L, al), dd = dep(D, ad), dr = dep(R, ar);
                                cur |= (lif == 0) & du ? kUp : 0u;
                                cur |= (lif == last) & dd ? kDn : 0u;
                                cur |= (jf == lstart) & dl ? kPrev : 0u;
                                cur |= (jf == lend - 1) & dr ? kNext : 0u;
                                if constexpr (!kSelective)   // feeds a node of the tile visited before it
                                    cur |= ((lif > 0) & du) | ((jf > lstart) & dl) ? kAgain : 0u;
                            }
                            // this lane leaves its tile
                            const bool leave = on & (jf == lend - 1);
                            prev = leave ? cur : prev;
                            cur = leave ? 0u : cur;
                            lstart = leave ? lend : lstart;
                            lend = leave ? min(nc, lend + T2J) : lend;
                            // slide the windows to step t + 1
                            um = nv; u0 = up; up = uq1; uq1 = uq2; uq2 = uq3;
                            if constexpr (!ADJ) { s0 = s1; s1 = s2; s2 = s3; s3 = s4; }
                            if constexpr (kSnap) { n0 = n1; n1 = n2; }
                            if constexpr (ADJ) {
                                tm = t0; t0 = tp; tp = tq1; tq1 = tq2; tq2 = tq3;
                                hu0 = hu1; hu1 = hu2; hu2 = hu3;
                                hd0 = hd1; hd1 = hd2; hd2 = hd3;
                            }
                        }
                        // ---- report the columns that every lane is through
                        if (lif == last && js + t - last > js) {
                            __threadfence_block();   // this lane wrote the row the strip downstream reads
                            s_prog[w] = pbase + min(js + t - last, endB);
                        }
                        if (t == doneA) {   // every lane is through tile cA
                            const int tt = tile_at(cA), tu = strip_tile(us, cA), td = strip_tile(ds, cA);
                            const unsigned f = __reduce_or_sync(0xffffffffu, lane_ok ? prev : 0u);
                            if (hasU) ok = wait_for(s_tdone + tu, o + 1);   // its marks on this tile have come
                            if (!ok) break;
                            if (lane == 0) {
                                int word_ = 0;
                                if constexpr (kSelective)
                                    word_ = (*(volatile int*)(s_dirty + tt) & 0xf & ~obit) | (int)(((f >> 8) & 0xf) << 4);
                                if (f & kChg) {
                                    word_ |= (f & kAgain) ? 0xf : (kSelective ? (0xf & ~obit) : 0);
                                    if ((f & kUp) && hasU) atomicOr(s_dirty + tu, 0xf);
                                    if ((f & kDn) && hasD) atomicOr(s_dirty + td, 0xf);
                                    if ((f & kPrev) && cA > 0) atomicOr(s_dirty + tile_at(cA - 1), 0xf);
                                    if ((f & kNext) && cA + 1 < nbj) atomicOr(s_dirty + tile_at(cA + 1), 0xf);
                                    if constexpr (kSnap) s_diff[tt] = (f & kMoved) ? 1 : 0;
                                    else if (f & kMoved) s_diff[tt] = 1;
                                }
                                *(volatile int*)(s_dirty + tt) = word_;
                            }
                            strip_publish(warp, s_tdone + tt, o + 1);
                            __syncwarp();
                            if (cB == cA) break;   // the stream ends here
                            cA = cB;
                            endA = endB;
                            firstA = firstB;
                            cornA = cornB;
                        }
                    }
                    cf = cB + 1;
                }
                __syncwarp();
            }
            __syncthreads();
            if (s_abort) break;   // block-uniform
            int any = 0, due_any = 0;
            for (int t = threadIdx.x; t < ntiles; t += nthr) {
                any |= s_diff[t];
                const int dm = s_dirty[t];
                due_any |= (kSelective ? (dm & (dm >> 4)) : dm) & 0xf;
            }
            any = __syncthreads_or(any);
            due_any = __syncthreads_or(due_any);
            ++it;
            if (!any) { moved_any = false; break; }
            // moved, but every tile locked: the next iteration would change nothing and pass the
            // test; it is counted without running
            if (!due_any && it < cap) { ++it; moved_any = false; break; }
        }
        if (threadIdx.x == 0) {
            result[q] = it | (moved_any ? 1 << 30 : 0);
            if (s_abort) atomicOr(queue + 1, 1);   // the host reports the stall
        }
        __syncthreads();
        if (s_abort) return;   // block-uniform
        __syncthreads();
    }
}

template <int KIND>
pfast_status launch_strips(const Sweep2Args& a, int nact, const int* caps, int* queue, int* result, cudaStream_t st) {
    int dev = 0, sms = 0, smem_max = 0, per_sm = 0;
    PFAST_CUDA_TRY(cudaGetDevice(&dev));
    PFAST_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PFAST_CUDA_TRY(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    PFAST_CUDA_TRY(cudaFuncSetAttribute(sweep2d_strips<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max - 256));
    const size_t smem = strips_smem<KIND>(a.nr, a.nc);
    PFAST_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sweep2d_strips<KIND>, a.nbi * 32, smem));
    const int blocks = std::min(nact, std::max(1, per_sm) * sms);
    sweep2d_strips<KIND><<<blocks, a.nbi * 32, smem, st>>>(a, nact, caps, queue, result);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "strip sweep launch", __FILE__, __LINE__);
    return PFAST_OK;
}

template <int KIND>
pfast_status launch_one2(const Sweep2Args& a, int d, int tiles, int nact, cudaStream_t st) {
    static bool attr_set = false;
    const size_t smem = (size_t)kWarps2 * warp_smem2<KIND>();
    if (!attr_set) {
        PFAST_CUDA_TRY(cudaFuncSetAttribute(sweep2d_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set = true;
    }
    dim3 grid((tiles + kWarps2 - 1) / kWarps2, nact);
    sweep2d_kernel<KIND><<<grid, kWarps2 * 32, smem, st>>>(a, d);
    return PFAST_OK;
}

constexpr int kThreads = 256;

__global__ void init2_kernel_d(double* base, const long long* off, const int* srcnode, long long n) {
    const int q = blockIdx.y;
    double* f = base + off[q];
    const int sn = srcnode[q];
    const long long s = sn >= 0 ? sn : -1;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        f[t] = (t == s) ? 0.0 : kInf;
}
__global__ void init2_kernel_f(float* base, const long long* off, const int* srcnode, long long n) {
    const int q = blockIdx.y;
    float* f = base + off[q];
    const int sn = srcnode[q];
    const long long s = sn >= 0 ? sn : -1;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        f[t] = (t == s) ? 0.0f : (float)kInf;
}

template <typename T>
__global__ void copy_inst_kernel(const T* a, T* b, const long long* oa, const long long* ob, long long n) {
    const int q = blockIdx.y;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        b[ob[q] + t] = a[oa[q] + t];
}

__global__ void widen_inst_kernel(const float* a, double* b, const long long* oa, const long long* ob, long long n) {
    const int q = blockIdx.y;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        b[ob[q] + t] = (double)a[oa[q] + t];
}

__global__ void narrow_inst_kernel(const double* a, float* b, const long long* oa, const long long* ob, long long n) {
    const int q = blockIdx.y;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        b[ob[q] + t] = (float)a[oa[q] + t];
}

__global__ void widen_lambda_inst_kernel(const float* a, double* b, const long long* oa, const long long* ob,
                                         const unsigned* mask, const long long* mo, int nr, int nc, int wpr) {
    const int q = blockIdx.y;
    const long long n = (long long)nr * nc;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const long long i = t / nc;
        const int j = (int)(t - i * nc);
        if (!((mask[mo[q] + i * wpr + (j >> 5)] >> (j & 31)) & 1u)) b[ob[q] + t] = (double)a[oa[q] + t];
    }
}

// One block per (source, reflector) instance: the reflection points of one reflector, then the
// INF reset above them.  The reference takes the columns in order, 1 .. nc-2, then 0, then nc-1
// (src/RT_pfsm2d.h:195,238,259), and each writes one node (k2+1, j) below its reflection row k2.
// Column j reads rows k2 and k2+1 of itself and of its neighbours j-1 and j+1, so of the columns
// before it it can meet only a neighbour's node, and only where that lies in row k2.  The
// columns are therefore evaluated together from the unchanged field, those that wait for a neighbour
// once it is done (chains as long as the reflector falls one row per column), and written at
// the end.  One thread per instance took 2.6 ms for 40 instances of 601 columns.
// v: the new values; state: 0 to do, 1 done, 2 no reflection point (both in shared memory).
__global__ void __launch_bounds__(256) reflect2_kernel(const Reflect2Args A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int q = blockIdx.x;
    double* U = A.U + A.inst_off[q];
    const int ir = A.inst_ir[q];
    const int nc = A.nc, nr = A.nr;
    const double dx = A.dx, dz = A.dz;
    const int* k2r = A.k2 + (long long)ir * nc;
    const int* qxc = A.qxcase + (long long)ir * nc;
    const double* Zr = A.Z + (long long)ir * nc * 3;
    double* v = reinterpret_cast<double*>(smem_raw);
    volatile unsigned char* state = smem_raw + sizeof(double) * nc;
    for (int j = threadIdx.x; j < nc; j += blockDim.x) state[j] = k2r[j] < 0 ? 2 : 0;   // 2: reflector below the model
    __syncthreads();
    // whether the reference takes column a before column b
    auto before = [&](int a, int b) {
        auto rank = [&](int j) { return j == nc - 1 ? nc + 1 : (j == 0 ? nc : j); };
        return rank(a) < rank(b);
    };
    for (;;) {   // each pass finishes at least the first unfinished column of the order
        int left = 0;
        for (int jj = threadIdx.x; jj < nc; jj += blockDim.x) {
            if (state[jj]) continue;
            const int k2 = k2r[jj], cs = qxc[jj];
            // the value of the neighbour column n in row k2 as the reference meets it
            bool ready = true;
            auto at = [&](int n) -> double {
                if (state[n] != 2 && before(n, jj) && k2r[n] + 1 == k2) {
                    if (state[n] == 1) { __threadfence_block(); return *(volatile double*)(v + n); }
                    ready = false;
                }
                return U[(long long)k2 * nc + n];
            };
            const double u0 = U[(long long)k2 * nc + jj];
            double qx;
            if (cs == 0) qx = (at(jj + 1) - at(jj - 1)) / 2.0 / dx;
            else if (cs == 1) qx = (u0 - at(jj - 1)) / dx;
            else qx = (at(jj + 1) - u0) / dx;
            if (!ready) { left = 1; continue; }
            const double qz = (U[(long long)(k2 + 1) * nc + jj] - u0) / dz;
            const double dnx = Zr[jj * 3 + 2], dnz = Zr[jj * 3 + 1], zd = Zr[jj * 3 + 0];
            const double rz = qz - 2 * (qx * dnx + qz * dnz) * dnz;
            const double r = u0 + qz * (zd - k2 * dz - dz) + rz * ((k2 + 1) * dz + dz - zd);
            *(volatile double*)(v + jj) = r;
            __threadfence_block();
            state[jj] = 1;
            if (r < 0) *A.err = 1;
        }
        if (!__syncthreads_or(left)) break;
    }
    for (int jj = threadIdx.x; jj < nc; jj += blockDim.x)
        if (state[jj] == 1) U[(long long)(k2r[jj] + 1) * nc + jj] = v[jj];
    __syncthreads();
    const int* kv = A.k2vec + (long long)ir * nc;
    for (int j = threadIdx.x; j < nc; j += blockDim.x) {
        const int top = min(kv[j], nr - 1);
        for (int i = 0; i <= top; ++i) U[(long long)i * nc + j] = kInf;
    }
}

// The same with one thread per instance, for more columns than shared memory holds.
__global__ void reflect2_serial_kernel(const Reflect2Args A, int ninst) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= ninst) return;
    double* U = A.U + A.inst_off[q];
    const int ir = A.inst_ir[q];
    const int nc = A.nc, nr = A.nr;
    const double dx = A.dx, dz = A.dz;
    const int* k2r = A.k2 + (long long)ir * nc;
    const int* qxc = A.qxcase + (long long)ir * nc;
    const double* Zr = A.Z + (long long)ir * nc * 3;
    for (int step = 0; step < nc; ++step) {
        // interior columns 1..nc-2 first, then column 0, then column nc-1 (src/RT_pfsm2d.h:195,238,259)
        const int jj = step < nc - 2 ? step + 1 : (step == nc - 2 ? 0 : nc - 1);
        const int k2 = k2r[jj];
        if (k2 < 0) continue;   // reflector below the model at this column: no reflection point
        double qx;
        const int cs = qxc[jj];
        if (cs == 0) qx = (U[(long long)k2 * nc + jj + 1] - U[(long long)k2 * nc + jj - 1]) / 2.0 / dx;
        else if (cs == 1) qx = (U[(long long)k2 * nc + jj] - U[(long long)k2 * nc + jj - 1]) / dx;
        else qx = (U[(long long)k2 * nc + jj + 1] - U[(long long)k2 * nc + jj]) / dx;
        const double u0 = U[(long long)k2 * nc + jj];
        const double qz = (U[(long long)(k2 + 1) * nc + jj] - u0) / dz;
        const double dnx = Zr[jj * 3 + 2], dnz = Zr[jj * 3 + 1], zd = Zr[jj * 3 + 0];
        const double rz = qz - 2 * (qx * dnx + qz * dnz) * dnz;
        const double v = u0 + qz * (zd - k2 * dz - dz) + rz * ((k2 + 1) * dz + dz - zd);
        U[(long long)(k2 + 1) * nc + jj] = v;
        if (v < 0) *A.err = 1;
    }
    for (int j = 0; j < nc; ++j) {
        const int kv = A.k2vec[(long long)ir * nc + j];
        for (int i = 0; i <= kv && i < nr; ++i) U[(long long)i * nc + j] = kInf;
    }
}

// One warp per instance: receiver boundary condition and misfit, rows in order.
__global__ void bc2_kernel(const Bc2Args A) {
    const int q = blockIdx.x, lane = threadIdx.x;
    const int s = A.inst_src[q], ir = A.inst_ir[q];
    const double* T = A.T + A.t_off[q];
    double* L = A.L + A.l_off[q];
    unsigned* mask = A.mask + A.mask_off[q];
    const int nc = A.nc, nr = A.nr;
    const int r0 = A.ch0[s], nrec = A.srnum[s];
    const int si = A.src_ij[2 * s], sj = A.src_ij[2 * s + 1];
    const bool trans = ir < 0;
    const double Cr = 1.0;
    double E = A.EE[q];   // running misfit: the reflection adjoint keeps one sum over all reflectors
    bool big = false;
    for (int base = 0; base < nrec; base += 32) {
        const int r = base + lane;
        double e = 0.0;
        if (r < nrec) {
            const int row = r0 + r;
            const double tob = trans ? A.ttobs[row] : A.trobs[(long long)row * A.numofr + ir];
            const bool picked = trans ? (tob < 100) : (tob != 0);
            if (picked) {
                const int i = A.rec[2 * row], j = A.rec[2 * row + 1];
                const long long o = (long long)i * nc + j;
                atomicOr(&mask[(long long)i * A.wpr + (j >> 5)], 1u << (j & 31));
                e = Cr * (tob - T[o]) * (tob - T[o]) / 2.0;
                const bool last = trans ? A.last_t[row] : A.last_r[(long long)row * A.numofr + ir];
                if (last && !(trans && i == si && j == sj)) {
                    const double ny = A.nxy[2 * row], nx = A.nxy[2 * row + 1];
                    const double Tz = (i + 1 >= nr) ? (T[o] - T[o - nc]) / A.dz : (T[o + nc] - T[o]) / A.dz;
                    const double Tx = (j + 1 >= nc) ? (T[o] - T[o - 1]) / A.dx : (T[o + 1] - T[o]) / A.dx;
                    double v = 0.0;
                    if (fabs(tob - T[o]) > 1e-9 && fabs(nx * Tx + ny * Tz) > 1e-6) v = Cr * (tob - T[o]) / (nx * Tx + ny * Tz);
                    L[o] = v;
                    if (fabs(v) > kConvTol) big = true;
                }
            }
        }
        for (int l = 0; l < 32; ++l) {
            const double el = __shfl_sync(0xffffffffu, e, l);
            if (lane == 0) E += el;
        }
    }
    big = __any_sync(0xffffffffu, big);
    if (lane == 0) {
        A.EE[q] = E;
        A.need[q] = big ? 1 : 0;
    }
}

__global__ void accumulate2_kernel(double* gT, double* gR, const double* lam, const long long* lo, const int* gslot,
                                   const double* vp, long long n, int ninst) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const double v = vp[t];
        const double v3 = v * v * v;
        double aT = gT[t], aR = gR[t];
        for (int q = 0; q < ninst; ++q) {
            const double x = lam[lo[q] + t] / v3;
            if (gslot[q] == 0) aT = aT - x;
            else aR = aR - x;
        }
        gT[t] = aT;
        gR[t] = aR;
    }
}

__global__ void blend2_kernel(const double* gT, const double* gR, const double* WR, double* gRT, long long n) {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        gRT[t] = gT[t] * (1. - WR[t]) + gR[t] * WR[t];   // src/RT_PFAST2D.cpp:434
}

__global__ void addto2_kernel(double* dst, const long long* dof, const double* src, const long long* sof, long long n) {
    const int q = blockIdx.y;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
        dst[dof[q] + t] = dst[dof[q] + t] + src[sof[q] + t];
}

__global__ void gather2_kernel(const double* fields, const long long* sfo, int numofr, long long n, const int* rec,
                               const int* ch0, const int* srnum, int b0, int nc, double* Tr) {
    const int b = blockIdx.y;
    const int s = b0 + b;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < srnum[s]; r += gridDim.x * blockDim.x) {
        const int row = ch0[s] + r;
        const long long o = (long long)rec[2 * row] * nc + rec[2 * row + 1];
        const double* base = fields + sfo[b];
        Tr[(long long)row * (numofr + 1)] = base[o];
        for (int ir = 0; ir < numofr; ++ir) Tr[(long long)row * (numofr + 1) + 1 + ir] = base[(1 + numofr + ir) * n + o];
    }
}

inline unsigned grid_for(long long n, int ninst) {
    long long b = (n + kThreads - 1) / kThreads;
    long long cap = std::max(1LL, 152LL * 16 / std::max(1, ninst) + 1);
    return (unsigned)std::max(1LL, std::min(b, cap));
}

}  // namespace

#define PFAST_LAUNCH_CHECK2()                                                                 \
    do {                                                                                      \
        cudaError_t e__ = cudaGetLastError();                                                 \
        if (e__ != cudaSuccess) return cuda_fail(e__, "kernel launch", __FILE__, __LINE__);   \
    } while (0)

pfast_status build_diag_table2(int nr, int nc, DiagTable2& t) {
    t.nbi = (nr + T2I - 1) / T2I;
    t.nbj = (nc + T2J - 1) / T2J;
    if (t.nbi > 65535 || t.nbj > 65535) {
        set_last_error("2D grid %dx%d too large", nr, nc);
        return PFAST_ERR_INVALID;
    }
    t.ndiag = t.nbi + t.nbj - 1;
    std::vector<unsigned> tiles;
    t.h_off.assign(t.ndiag + 1, 0);
    for (int d = 0; d < t.ndiag; ++d) {
        t.h_off[d] = (int)tiles.size();
        for (int bi = 0; bi < t.nbi; ++bi) {
            const int bj = d - bi;
            if (bj >= 0 && bj < t.nbj) tiles.push_back((unsigned)bi | ((unsigned)bj << 16));
        }
    }
    t.h_off[t.ndiag] = (int)tiles.size();
    PFAST_CUDA_TRY(cudaMalloc(&t.d_off, sizeof(int) * t.h_off.size()));
    PFAST_CUDA_TRY(cudaMalloc(&t.d_tiles, sizeof(unsigned) * tiles.size()));
    PFAST_CUDA_TRY(cudaMemcpy(t.d_off, t.h_off.data(), sizeof(int) * t.h_off.size(), cudaMemcpyHostToDevice));
    PFAST_CUDA_TRY(cudaMemcpy(t.d_tiles, tiles.data(), sizeof(unsigned) * tiles.size(), cudaMemcpyHostToDevice));
    return PFAST_OK;
}

void free_diag_table2(DiagTable2& t) {
    if (t.d_off) cudaFree(t.d_off);
    if (t.d_tiles) cudaFree(t.d_tiles);
    t.d_off = nullptr;
    t.d_tiles = nullptr;
}

template <typename Real>
__global__ void near_source2_kernel(Real* __restrict__ base, const long long* __restrict__ off,
                                    const int* __restrict__ inst_src, const int* __restrict__ inst_lim,
                                    const int* __restrict__ rowlim, const double* __restrict__ s64, int nr, int nc,
                                    double dx, double dz, int r) {
    const int q = blockIdx.y;
    if (inst_src[q] < 0) return;
    const int si = inst_src[q] >> 16, sj = inst_src[q] & 0xffff;
    const int* rl = inst_lim[q] >= 0 ? rowlim + (long long)inst_lim[q] * nc : nullptr;
    const double ss = s64[(long long)si * nc + sj];
    const int w = 2 * r + 1;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < w * w; t += gridDim.x * blockDim.x) {
        const int qi = t / w - r, qj = t % w - r;
        const int i = si + qi, j = sj + qj;
        if (i < 0 || i >= nr || j < 0 || j >= nc || qi * qi + qj * qj > r * r) continue;
        if (rl != nullptr && i > rl[j]) continue;   // below the reflector: not part of this solve
        const long long node = (long long)i * nc + j;
        const double ez = qi * dz, ex = qj * dx;
        base[off[q] + node] = Real(0.5 * (ss + s64[node]) * sqrt(ez * ez + ex * ex));
    }
}

pfast_status launch_near_source2(void* base, int is_fp32, const long long* off, const int* inst_src,
                                 const int* inst_lim, const int* rowlim, const double* s64, int nr, int nc, double dx,
                                 double dz, int radius, int ninst, cudaStream_t st) {
    if (radius <= 0 || ninst <= 0) return PFAST_OK;
    const int w = 2 * radius + 1;
    dim3 grid((unsigned)std::max(1, (w * w + 255) / 256), ninst);
    if (is_fp32)
        near_source2_kernel<float><<<grid, 256, 0, st>>>((float*)base, off, inst_src, inst_lim, rowlim, s64, nr, nc, dx,
                                                         dz, radius);
    else
        near_source2_kernel<double><<<grid, 256, 0, st>>>((double*)base, off, inst_src, inst_lim, rowlim, s64, nr, nc,
                                                          dx, dz, radius);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "near_source2 launch", __FILE__, __LINE__);
    return PFAST_OK;
}

pfast_status launch_seed_tiles2(int kind, const Sweep2Args& a, int nact, cudaStream_t st) {
    if (nact <= 0) return PFAST_OK;
    dim3 grid((unsigned)((a.ntiles + 7) / 8), nact);
    switch (kind) {
        case kFwdPlain64: seed_tiles2_kernel<double, false, false><<<grid, 256, 0, st>>>(a); break;
        case kAdjPlain64: seed_tiles2_kernel<double, true, false><<<grid, 256, 0, st>>>(a); break;
        case kFwdFast32: seed_tiles2_kernel<float, false, false><<<grid, 256, 0, st>>>(a); break;
        case kAdjFast32: seed_tiles2_kernel<float, true, false><<<grid, 256, 0, st>>>(a); break;
        case kAdjPolish64: seed_tiles2_kernel<double, true, true><<<grid, 256, 0, st>>>(a); break;
        default: return PFAST_OK;
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "seed tiles2 launch", __FILE__, __LINE__);
    return PFAST_OK;
}

pfast_status launch_sweep2(int kind, const Sweep2Args& a, int d, int tiles, int nact, cudaStream_t st) {
    if (tiles <= 0 || nact <= 0) return PFAST_OK;
    switch (kind) {
        case kFwdPlain64: return launch_one2<kFwdPlain64>(a, d, tiles, nact, st);
        case kFwdFast32: return launch_one2<kFwdFast32>(a, d, tiles, nact, st);
        case kFwdPolish64: return launch_one2<kFwdPolish64>(a, d, tiles, nact, st);
        case kAdjPlain64: return launch_one2<kAdjPlain64>(a, d, tiles, nact, st);
        case kAdjFast32: return launch_one2<kAdjFast32>(a, d, tiles, nact, st);
        case kAdjPolish64: return launch_one2<kAdjPolish64>(a, d, tiles, nact, st);
    }
    set_last_error("unknown sweep kind %d", kind);
    return PFAST_ERR_INVALID;
}

pfast_status launch_split_inst(const double* a, void* b, const long long* oa, const long long* ob, long long n, int ninst,
                               cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    dim3 grid(grid_for(n, ninst), ninst);
    split_inst_kernel<<<grid, kThreads, 0, st>>>(a, (float2*)b, oa, ob, n);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

// Grids the strips schedule takes: a block's warps and shared memory.
bool strips_fit(int kind, int nr, int nc) {
    const bool f32 = kind == kFwdFast32 || kind == kAdjFast32;
    const size_t smem = f32 ? strips_smem<kFwdFast32>(nr, nc) : strips_smem<kFwdPlain64>(nr, nc);
    return (nr + T2I - 1) / T2I <= kStripMax && smem <= 200 * 1024;
}

pfast_status launch_sweep2_strips(int kind, const Sweep2Args& a, int nact, const int* caps, int* queue, int* result,
                                  cudaStream_t st) {
    if (nact <= 0) return PFAST_OK;
    switch (kind) {
        case kFwdPlain64: return launch_strips<kFwdPlain64>(a, nact, caps, queue, result, st);
        case kFwdFast32: return launch_strips<kFwdFast32>(a, nact, caps, queue, result, st);
        case kFwdPolish64: return launch_strips<kFwdPolish64>(a, nact, caps, queue, result, st);
        case kAdjPlain64: return launch_strips<kAdjPlain64>(a, nact, caps, queue, result, st);
        case kAdjFast32: return launch_strips<kAdjFast32>(a, nact, caps, queue, result, st);
        case kAdjPolish64: return launch_strips<kAdjPolish64>(a, nact, caps, queue, result, st);
    }
    set_last_error("unknown sweep kind %d", kind);
    return PFAST_ERR_INVALID;
}

pfast_status launch_init2(void* base, int is_fp32, const long long* off, const int* srcnode, long long n, int ninst,
                          cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    dim3 grid(grid_for(n, ninst), ninst);
    if (is_fp32) init2_kernel_f<<<grid, kThreads, 0, st>>>((float*)base, off, srcnode, n);
    else init2_kernel_d<<<grid, kThreads, 0, st>>>((double*)base, off, srcnode, n);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_copy_inst(const void* src, void* dst, int is_fp32, const long long* os, const long long* od,
                              long long n, int ninst, cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    dim3 grid(grid_for(n, ninst), ninst);
    if (is_fp32) copy_inst_kernel<float><<<grid, kThreads, 0, st>>>((const float*)src, (float*)dst, os, od, n);
    else copy_inst_kernel<double><<<grid, kThreads, 0, st>>>((const double*)src, (double*)dst, os, od, n);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_widen_inst(const float* a, double* b, const long long* oa, const long long* ob, long long n,
                               int ninst, cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    dim3 grid(grid_for(n, ninst), ninst);
    widen_inst_kernel<<<grid, kThreads, 0, st>>>(a, b, oa, ob, n);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_narrow_inst(const double* a, float* b, const long long* oa, const long long* ob, long long n,
                                int ninst, cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    dim3 grid(grid_for(n, ninst), ninst);
    narrow_inst_kernel<<<grid, kThreads, 0, st>>>(a, b, oa, ob, n);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_widen_lambda_inst(const float* a, double* b, const long long* oa, const long long* ob,
                                      const unsigned* mask, const long long* mo, int nr, int nc, int wpr, int ninst,
                                      cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    dim3 grid(grid_for((long long)nr * nc, ninst), ninst);
    widen_lambda_inst_kernel<<<grid, kThreads, 0, st>>>(a, b, oa, ob, mask, mo, nr, nc, wpr);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_reflect2(const Reflect2Args& a, int ninst, cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    const size_t smem = 9 * (size_t)a.nc;
    if (smem <= 48 * 1024) reflect2_kernel<<<ninst, 256, smem, st>>>(a);
    else reflect2_serial_kernel<<<(ninst + 63) / 64, 64, 0, st>>>(a, ninst);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_bc2(const Bc2Args& a, int ninst, cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    bc2_kernel<<<ninst, 32, 0, st>>>(a);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_accumulate2(double* gT, double* gR, const double* lam, const long long* lo, const int* gslot,
                                const double* vp, long long n, int ninst, cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    accumulate2_kernel<<<grid_for(n, 1), kThreads, 0, st>>>(gT, gR, lam, lo, gslot, vp, n, ninst);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_blend2(const double* gT, const double* gR, const double* WR, double* gRT, long long n,
                           cudaStream_t st) {
    blend2_kernel<<<grid_for(n, 1), kThreads, 0, st>>>(gT, gR, WR, gRT, n);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_addto2(double* dst, const long long* dof, const double* src, const long long* sof, long long n,
                           int ninst, cudaStream_t st) {
    if (ninst <= 0) return PFAST_OK;
    dim3 grid(grid_for(n, ninst), ninst);
    addto2_kernel<<<grid, kThreads, 0, st>>>(dst, dof, src, sof, n);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

pfast_status launch_gather2(const double* fields, const long long* sfo, int numofr, long long n, const int* rec,
                            const int* ch0, const int* srnum, int nbatch, int b0, int nc, double* Tr, cudaStream_t st) {
    if (nbatch <= 0) return PFAST_OK;
    dim3 grid(8, nbatch);
    gather2_kernel<<<grid, kThreads, 0, st>>>(fields, sfo, numofr, n, rec, ch0, srnum, b0, nc, Tr);
    PFAST_LAUNCH_CHECK2();
    return PFAST_OK;
}

}  // namespace pfast
