// exact_arith.h -- the plain FP64 node updates with fewer FP64 instructions and the same bits
// (host and device code; the CPU check tests/native/exact_arith_check.cpp compiles it with g++).
//
// What bounds the plain sweeps is the FP64 pipe: on this part an FP64 warp instruction holds its
// SM sub-partition for 64 cycles (measured: one warp, dependent or independent; 76 with all four
// sub-partitions busy), and an FP64 division costs 8 to 9 such instructions, a square root 10.
// The reference's 3D Godunov update (src/T_pfsm3d.h:99-119) holds 13 divisions by constants of the
// grid and 2 square roots, its adjoint update (src/T_padjoint3d.h:42-71) 12 and one by a variable.
// So
//   * a division by a grid constant d multiplies by its reciprocal as an unevaluated sum
//     rh + rl (rh = 1/d rounded, rl = the remainder, rounded): q = fma(x, rh, t), t = x * rl.  x / d is
//     at least 2^-(54+m) relative away from every rounding boundary when the odd part of d's
//     significand has m bits, and |t| <= 2^-53 |q|, so t in FP32 (2^-22 relative) leaves q correctly
//     rounded whenever m <= 18, and t in FP64 whenever m <= 48 (Brisebarre, Muller and Raina,
//     "Accelerating correctly rounded floating-point division when the divisor is known in
//     advance", IEEE Trans. Comput. 53(8), 2004).  For other d one more step, r = fma(-d, q, x)
//     and fma(r, rh, q), is correctly rounded because q is faithful (P. Markstein, "Computation
//     of elementary functions on the IBM RISC System/6000 processor", 1990).  1 FP64 instruction
//     (3 for long d) instead of 8 to 9; the FP32 and integer ones run beside the FP64 pipe.
//   * a square root refines an FP32 reciprocal root twice (Newton), and is rounded by the sign of the
//     exact remainder against half an ulp: 6 FP64 instructions instead of about 10.
//   * scalings by powers of two are left out where they commute with rounding, terms the reference
//     multiplies by +0 are not formed, and POS / NEG are taken from the sign bit.
//   * the branch of the reference's case analysis that a node takes is predicted from FP32 copies
//     with a margin far above every rounding error, so that a 3-neighbour node does not evaluate
//     the 2-neighbour solution first.
// Arguments outside the exponent range in which these identities hold take the reference's
// expressions as they stand.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef PFAST_HD
#ifdef __CUDACC__
#define PFAST_HD __host__ __device__ __forceinline__
#else
#define PFAST_HD inline
#endif
#endif

namespace pfast {

// The reference's "infinity" for unreached nodes (INF macro, src/T_pfsm3d.h:12-14).
constexpr double kUnreached = 9999999.0;

PFAST_HD long long bits_of(double x) {
#ifdef __CUDA_ARCH__
    return __double_as_longlong(x);
#else
    long long b;
    std::memcpy(&b, &x, sizeof(b));
    return b;
#endif
}
PFAST_HD double from_bits(long long b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double(b);
#else
    double x;
    std::memcpy(&x, &b, sizeof(x));
    return x;
#endif
}
PFAST_HD int exponent_of(double x) { return (int)((unsigned long long)bits_of(x) >> 52) & 0x7ff; }
PFAST_HD bool is_zero(double x) { return ((unsigned long long)bits_of(x) << 1) == 0; }

// An integer that orders like the value (NaNs beyond the infinities).
PFAST_HD long long ordered(double x) {
    const long long b = bits_of(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}

// A divisor known in advance, in [2^-41, 2^42].
struct DivBy {
    double d, rh, rl;
    float rl60;    // rl * 2^60 as FP32 (so that x * rl60 stays in its range for |x| in [2^-90, 2^90])
    int fast;      // m <= 18: q = fma(x, rh, t) with t in FP32 is correctly rounded
    int short_;    // m <= 48: the same with t in FP64
    int emin;      // biased exponent from which t in FP64 (and for long d the remainder) loses no bit
};

// Host: the constants of a positive normal divisor.
inline DivBy div_by(double d) {
    DivBy k;
    k.d = d;
    k.rh = 1.0 / d;
    k.rl = std::fma(-d, k.rh, 1.0) / d;   // the remainder 1 - d rh is exact
    k.rl60 = (float)std::ldexp(k.rl, 60);
    unsigned long long m = ((unsigned long long)bits_of(d) & 0xfffffffffffffull) | (1ull << 52);
    while (!(m & 1)) m >>= 1;
    k.fast = m < (1ull << 18);
    k.short_ = m < (1ull << 48);
    // t rounds to a multiple of 2^-1074: with m <= 48 that is below 2^-(54+m) |q| from |q| >= 2^-960 on;
    // the remainder of long d is a multiple of 2^-104 |x|
    k.emin = 1023 - 950 + (d > 1.0 ? std::ilogb(d) : 0);
    return k;
}

// FP32 <-> FP64 on the integer pipe, for magnitudes in [2^-120, 2^120] (an FP32 zero becomes 2^-187 or
// so, far below half an ulp of what it is added to).
PFAST_HD float cut32(double x) {   // truncated
    const unsigned hi = (unsigned)((unsigned long long)bits_of(x) >> 32), lo = (unsigned)bits_of(x);
    const unsigned u = (hi & 0x80000000u) | ((((hi & 0x7fffffffu) - (896u << 20)) << 3) | (lo >> 29));
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, sizeof(f));
    return f;
#endif
}
template <int SHIFT>   // x * 2^-SHIFT
PFAST_HD double wide64(float x) {
    unsigned u;
#ifdef __CUDA_ARCH__
    u = __float_as_uint(x);
#else
    std::memcpy(&u, &x, sizeof(u));
#endif
    const unsigned mag = u & 0x7fffffffu;
    const unsigned hi = (u & 0x80000000u) | ((mag >> 3) + ((896u - SHIFT) << 20));
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)(mag << 29));
#else
    return from_bits((long long)(((unsigned long long)hi << 32) | (unsigned)(mag << 29)));
#endif
}

// x / d for x in +-[2^-90, 2^90]: FAST for divisors with fast set, else any.
template <bool FAST>
PFAST_HD double div_exact(double x, double d, double rh, float rl60) {
    const double q = fma(x, rh, wide64<60>(cut32(x) * rl60));
    return FAST ? q : fma(fma(-d, q, x), rh, q);
}
template <bool FAST>
PFAST_HD double div_exact(double x, const DivBy& k) { return div_exact<FAST>(x, k.d, k.rh, k.rl60); }

// A value the compiler may not compute with ahead of the branch it is used in.
PFAST_HD double here(double x) {
#ifdef __CUDA_ARCH__
    asm volatile("" : "+d"(x));
#endif
    return x;
}
// x / k.d for any x: zeros keep their sign, the ends of the exponent range divide.
PFAST_HD double div_any(double x, const DivBy& k) {
    const int e = exponent_of(x);
    double q = fma(x, k.rh, x * k.rl);
    if (!k.short_) q = fma(fma(-k.d, q, x), k.rh, q);
    if (is_zero(x)) q = x;
    else if ((unsigned)(e - k.emin) > (unsigned)(1923 - k.emin)) q = here(x) / k.d;   // tiny, > 2^900, inf or NaN
    return q;
}
// The same for arguments that are as a rule zero or in [2^-90, 2^90] (traveltime differences).
PFAST_HD double div_mid(double x, const DivBy& k) {
    double q = fma(x, k.rh, wide64<60>(cut32(x) * k.rl60));
    if (!k.fast) q = fma(fma(-k.d, q, x), k.rh, q);
    if (is_zero(x)) q = x;
    else if ((unsigned)(exponent_of(x) - 933) > 180u) q = here(x) / k.d;
    return q;
}

// sqrt(x), correctly rounded, for x >= +0.  With y = 1/sqrt(x) to 2^-21, g = x y and two Newton steps
// g += (x - g^2) y / 2 leave g within 2^-62 relative before the last rounding, so g is one of the
// two neighbours of the root.  The remainder r = x - g^2 is then exact, and root > g + u/2 exactly
// where r > g u, root < g - u/2 where r <= -g u (u: ulp of g; both sides are multiples of u^2, and the
// root of an FP64 number is never a midpoint); below a power of two the spacing halves, and any
// negative remainder means the next number down.
#ifndef __CUDACC__
inline float g_seed_error = 1.0f;   // the CPU check spreads the seed's error
#endif
PFAST_HD double sqrt_exact(double x) {
    if ((unsigned)(exponent_of(x) - 923) > 200u) return sqrt(here(x));   // outside 2^+-100 (zero, inf among them)
    const float xf = cut32(x);
    float yf;
#ifdef __CUDA_ARCH__
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(xf));
#elif defined(__CUDACC__)
    yf = 1.0f / sqrtf(xf);
#else
    yf = g_seed_error / sqrtf(xf);
#endif
    const double y = wide64<0>(yf), h = wide64<1>(yf);
    double g = x * y;
    g = fma(fma(-g, g, x), h, g);
    g = fma(fma(-g, g, x), h, g);
    const double r = fma(-g, g, x);
    const long long gb = bits_of(g);
    const double gu = from_bits(gb + ((long long)(exponent_of(g) - 1023 - 52) << 52));   // g * ulp(g)
    const bool low = (gb & 0xfffffffffffffll) == 0 ? bits_of(r) < 0 && !is_zero(r) : ordered(r) <= ordered(-gu);
    return from_bits(gb + (ordered(r) > bits_of(gu) ? 1 : 0) - (low ? 1 : 0));
}

// Grid constants of the exact updates.
struct ExactGrid3 {
    DivBy axis[3];     // d of x, y, z
    DivBy pair[3];     // d*d of the two other axes, summed: pair[a] leaves axis a out
    DivBy all[3];      // 1/d^2 summed with axis a last (the reference adds the smallest neighbour's axis last)
    double dd[3];      // d*d
    double d4;         // ((d*d)*d)*d of axis x
    int iso;           // one spacing
    int fast;          // the spacings divide in one FP64 instruction
    int quick;         // the spacings lie in the range the identities need
};

inline ExactGrid3 exact_grid3(const double d[3]) {
    ExactGrid3 g;
    std::memset(&g, 0, sizeof(g));
    g.quick = 1;
    for (int a = 0; a < 3; ++a) {
        if (!(d[a] > 0x1p-20 && d[a] < 0x1p20)) g.quick = 0;
    }
    if (!g.quick) return g;
    g.fast = 1;
    double inv2[3];
    for (int a = 0; a < 3; ++a) {
        g.axis[a] = div_by(d[a]);
        g.fast &= g.axis[a].fast;
        g.dd[a] = d[a] * d[a];
        inv2[a] = 1.0 / d[a] / d[a];
    }
    for (int a = 0; a < 3; ++a) {
        const int p = (a + 1) % 3, q = (a + 2) % 3;
        g.pair[a] = div_by(g.dd[p] + g.dd[q]);
        g.all[a] = div_by((inv2[p] + inv2[q]) + inv2[a]);
    }
    g.d4 = g.dd[0] * d[0] * d[0];
    g.iso = d[0] == d[1] && d[1] == d[2];
    return g;
}

// |v| in [2^-34, 2^34]: traveltimes for which every quotient above stays in its range
PFAST_HD bool in_range(double v) { return (unsigned)(exponent_of(v) - 989) <= 67u; }
// Slownesses below 2^58 as well (the root of the terms with s*s is then below 2^119): where those overflow
// (from about 2^450 on, velocities below 1e-136 of an impermeable body) the one-step quotient of an
// infinite numerator is NaN, where x / d is infinite and the minimum with the node's value drops it.
PFAST_HD bool slow_in_range(double s) { return exponent_of(s) <= 1080; }

// Magnitude of a value >= +0 as FP32 (truncated; +inf and beyond give a huge finite value).
PFAST_HD float approx32(double v) {
    const unsigned hi = (unsigned)((unsigned long long)bits_of(v) >> 32), lo = (unsigned)bits_of(v);
    unsigned u = 0;
    if (hi >= (1151u << 20)) u = 0x7f000000u;
    else if (hi >= (897u << 20)) u = ((hi - (896u << 20)) << 3) | (lo >> 29);
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, sizeof(f));
    return f;
#endif
}

// The reference's expressions as they stand: sorted neighbour minima a >= b >= c with their
// spacings and 1/d^2, the 1-neighbour value already found above b.
PFAST_HD double eik3_tail_ref(double a, double b, double c, double da, double db, double dc, double ia, double ib,
                              double ic, double s) {
    double A = dc * dc + db * db;
    double B = -2. * (b * dc * dc + c * db * db);
    double C = dc * dc * b * b + db * db * c * c - db * db * dc * dc * s * s;
    double D = B * B - 4. * A * C;
    double q = (D >= 0) ? (-B + sqrt(D)) / 2. / A : kUnreached;
    if (bits_of(q) <= bits_of(a)) return q;
    A = ia + ib + ic;
    B = -2.0 * (a / da / da + b / db / db + c / dc / dc);
    C = a * a / da / da + b * b / db / db + c * c / dc / dc - s * s;
    D = B * B - 4. * A * C;
    q = (D >= 0) ? (-B + sqrt(D)) / 2. / A : kUnreached;
    return q;
}

// The reference's 3D Godunov solution (src/T_pfsm3d.h:99-119) for neighbour minima x, y, z along
// the axes and slowness s, bit for bit.  With S = -B/2 and D = 4 (S*S - A*C) the factors 2 and 4
// are exact and left out.  The 2- and the 3-neighbour solution share the square root and the
// division: per warp at most 2 + 13 + 21 + 13 FP64 instructions (spacings of few bits), where the
// expressions as they stand take about 185.  96 x 96 x 48 nodes, 16 sources, one launch per tile
// diagonal: forward sweeps 210 -> 140 ms with FP64 tails and the library's root.
// MIN: only the minimum with a node's value (at most the unreached one) counts, so that for a slowness
// out of range, whose solutions are all 2^37 or more (spacings above 2^-20), any larger value does: a body
// that lets nothing through does not run the expressions beside the other lanes' short form.
template <bool ISO, bool FAST, bool MIN = false>
PFAST_HD double eik3_exact(double x, double y, double z, double s, const ExactGrid3& g, const double* inv2) {
    double a = x, b = y, c = z, t;
    int ka = 0, kb = 1, kc = 2, k;
    if (bits_of(b) > bits_of(a)) { t = a; a = b; b = t; k = ka; ka = kb; kb = k; }
    if (bits_of(c) > bits_of(a)) { t = a; a = c; c = t; k = ka; ka = kc; kc = k; }
    if (bits_of(c) > bits_of(b)) { t = b; b = c; c = t; k = kb; kb = kc; kc = k; }
    auto pick = [](int i, double v0, double v1, double v2) { return ISO ? v0 : (i == 0 ? v0 : (i == 1 ? v1 : v2)); };
    const double dc = pick(kc, g.axis[0].d, g.axis[1].d, g.axis[2].d);
    double q = dc * s + c;
    if (bits_of(q) <= bits_of(b)) return q;
    const double db = pick(kb, g.axis[0].d, g.axis[1].d, g.axis[2].d);
    const bool ainf = bits_of(a) >= 0x7ff0000000000000ll;
    if (!(in_range(b) && (is_zero(c) || in_range(c)) && (ainf || in_range(a)) && slow_in_range(s))) {
        if (MIN && !slow_in_range(s)) return INFINITY;
        const double da = pick(ka, g.axis[0].d, g.axis[1].d, g.axis[2].d);
        return eik3_tail_ref(a, b, c, da, db, dc, pick(ka, inv2[0], inv2[1], inv2[2]),
                             pick(kb, inv2[0], inv2[1], inv2[2]), pick(kc, inv2[0], inv2[1], inv2[2]), s);
    }
    // Three neighbours for certain: the 2-neighbour solution exceeds a exactly where
    // (a-b)^2/db^2 + (a-c)^2/dc^2 < s^2.  FP32 differences of truncated copies err by at most
    // 2^-22 a; that is held below 1 % of the 1-neighbour step, where the FP64 formulas are
    // accurate to 1e-6 of it, and the test asks for 2 %.  Anything closer evaluates both, in the
    // reference's order.
    bool three;
    {
        const float af = approx32(a), bf = approx32(b), cf = approx32(c), sf = approx32(s);
        const float err = af * 2.4e-7f;
        const float fb = (af - bf) + err, fc = (af - cf) + err;
        const float hb = ISO ? 0.0f : approx32(db), hc = approx32(dc);
        const float stepc = hc * sf, stepb = ISO ? stepc : hb * sf;   // 1-neighbour steps along the two axes
        const float lo = stepc < stepb ? stepc : stepb;
        // (fb / stepb)^2 + (fc / stepc)^2 < 0.98
        three = err <= 0.01f * lo && fb * fb * (stepc * stepc) + fc * fc * (stepb * stepb) <
                                         0.98f * (stepb * stepb) * (stepc * stepc) && lo > 1e-8f && af < 1e8f;
    }
    for (;;) {
        double S, C, A, Ah;
        float Al;
        auto pickf = [](int i, float v0, float v1, float v2) { return ISO ? v0 : (i == 0 ? v0 : (i == 1 ? v1 : v2)); };
        if (three) {
            auto dv = [&](double v, int i) {
                return div_exact<FAST>(v, pick(i, g.axis[0].d, g.axis[1].d, g.axis[2].d),
                                       pick(i, g.axis[0].rh, g.axis[1].rh, g.axis[2].rh),
                                       pickf(i, g.axis[0].rl60, g.axis[1].rl60, g.axis[2].rl60));
            };
            // c = 0 at the neighbours of the source
            auto dv0 = [&](double v, int i) { const double r = dv(v, i); return is_zero(v) ? v : r; };
            S = dv(dv(a, ka), ka) + dv(dv(b, kb), kb) + dv0(dv0(c, kc), kc);
            C = dv(dv(a * a, ka), ka) + dv(dv(b * b, kb), kb) + dv0(dv0(c * c, kc), kc) - s * s;
            A = pick(kc, g.all[0].d, g.all[1].d, g.all[2].d);
            Ah = pick(kc, g.all[0].rh, g.all[1].rh, g.all[2].rh);
            Al = pickf(kc, g.all[0].rl60, g.all[1].rl60, g.all[2].rl60);
        } else {
            const double ddc = pick(kc, g.dd[0], g.dd[1], g.dd[2]), ddb = pick(kb, g.dd[0], g.dd[1], g.dd[2]);
            S = b * dc * dc + c * db * db;
            C = ddc * b * b + ddb * c * c - (ISO ? g.d4 : ddb * dc * dc) * s * s;
            A = pick(ka, g.pair[0].d, g.pair[1].d, g.pair[2].d);
            Ah = pick(ka, g.pair[0].rh, g.pair[1].rh, g.pair[2].rh);
            Al = pickf(ka, g.pair[0].rl60, g.pair[1].rl60, g.pair[2].rl60);
        }
        const double D = S * S - A * C;
        q = (D >= 0) ? div_exact<false>(S + sqrt_exact(D), A, Ah, Al) : kUnreached;
        if (three || bits_of(q) <= bits_of(a)) return q;
        three = true;
    }
}

// The reference's 3D adjoint update (src/T_padjoint3d.h:42-71), bit for bit, for reached
// traveltimes (the caller returns 0 next to an unreached one).  Per axis at most one of the two
// POS / NEG terms of a difference pair is nonzero except at a local extremum of T, so one product
// and no subtraction remain there.  40 to 50 FP64 instructions (spacings of few bits) instead of
// about 150.
PFAST_HD double pos_part(double x) { return bits_of(x) > 0 ? x : 0.0; }                  // (x + |x|) / 2
PFAST_HD double neg_part(double x) { return bits_of(x) < 0 ? x : 0.0; }                  // (x - |x|) / 2
// p - m with one of the two zero (any signs): no FP64 instruction unless both are nonzero or both zero.
PFAST_HD double sub_sparse(double p, double m) {
    const bool zp = is_zero(p), zm = is_zero(m);
    if (zp == zm) return p - m;
    return zm ? p : from_bits(bits_of(m) ^ (long long)0x8000000000000000ull);
}
// Whether they hold for traveltimes whose upper words are at most `most` as unsigned numbers (below the
// unreached value that is: no NaN, -inf or value below -2^999, whose x + |x| overflows or is NaN).
// Once per node: tested per axis, the adjoint of 16 shots of 96 x 96 x 48 took 148.6 ms per diagonal, 145.6 so.
PFAST_HD unsigned upper_of(double x) { return (unsigned)((unsigned long long)bits_of(x) >> 32); }
PFAST_HD unsigned most_of(unsigned a, unsigned b) { return a > b ? a : b; }
PFAST_HD bool adj_ordinary(unsigned most) { return most < 0xfe600000u; }
// One axis: den += ..., num += ... of the reference, g.. as its POS / NEG arguments.
PFAST_HD void adj_axis_exact(double T0, double Tp, double Tm, double Lp, double Lm, const DivBy& k, double& den,
                             double& num) {
    const double gp = div_mid(-(Tp - T0), k), gm = div_mid(-(T0 - Tm), k);
    const double pp = pos_part(gp), nm = neg_part(gm), pm = pos_part(gm), np = neg_part(gp);
    den = div_mid(sub_sparse(pp, nm), k);
    // pm * Lm - np * Lp
    const bool zpm = is_zero(pm), znp = is_zero(np);
    double n;
    if (zpm != znp) {
        const double co = zpm ? np : pm, L = zpm ? Lp : Lm;   // the other product is a zero
        double v = co * L;
        if (zpm) v = from_bits(bits_of(v) ^ (long long)0x8000000000000000ull);
        // a zero or non-finite result depends on the other term too: the expression as it stands
        n = is_zero(v) || exponent_of(Lp) == 0x7ff || exponent_of(Lm) == 0x7ff ? pm * Lm - np * Lp : v;
    } else {
        n = pm * Lm - np * Lp;
    }
    num = div_any(n, k);
}

// Whether the plain 3D forward update of a node of value vn can change in any bit when a neighbour's value
// changes, lo being forward_change of its two values.  The formula is exact to within
// sqrt(k eps) = 4e-8 relative to its largest argument at worst (its discriminant cancels), so a
// neighbour 2^-20 relative above the node can neither lower the minimum of the node's value and the
// formula's nor take part in it -- unless the discriminant of the 2-neighbour solution rounds below 0,
// upon which the reference goes on to the third neighbour whatever its value.  Its exact value is
// at least db^4 dc^2 s^2 where that solution is asked for (1-neighbour value dc s + c above b) and dmax <=
// 512 dmin, its rounding error below k eps ((dc^2 + db^2) b)^2, so it stays positive from
// s dmin^2 / (2 dmax) >= 2^-20 b on, k up to 2000; with b < vn (1 + 2^-20) + dmax s, for vn <= s dmin^2 /
// dmax 2^17.  A change above that (forward_prune_limit with the model's least slowness: 131072 steps on an
// equally spaced grid) counts for every neighbour (a neighbour that is spared lies below the change).
inline int forward_prune_limit(const double d[3], double vmax) {
    const double lo = std::fmin(d[0], std::fmin(d[1], d[2])), hi = std::fmax(d[0], std::fmax(d[1], d[2]));
    const double t = lo * (lo / hi) / vmax * 0x1p17;
    // the upper word of t rounded down to a power of two, so that models of an inversion share the
    // captured launches; 0: no bound holds
    return hi <= 512.0 * lo && t > 0x1p-1000 && t < 0x1p1000 ? (1023 + std::ilogb(t)) << 20 : 0;
}
// The bits of the smaller value, or of less than every number (limit_hi: the upper word of the limit, whose
// lower one is 0: tested per neighbour and in 64 bits, the one-shot solves took 5 % longer).
PFAST_HD long long forward_change(double old, double nv, int limit_hi) {
    const long long a = bits_of(old), b = bits_of(nv), lo = a < b ? a : b;
    const int hi = (int)(lo >> 32);
    return ((long long)(hi >= limit_hi ? (int)0x80000000 : hi) << 32) | (unsigned)lo;
}
PFAST_HD bool forward_depends_exact(long long lo, double vn) { return lo < bits_of(vn) + (1ll << 33); }
// Whether the plain adjoint update of a node (traveltime tn, value vn) can change in any bit when its
// neighbour of traveltime t0 goes from `old` to `nv`.  A neighbour of smaller or equal traveltime
// enters as +0 * lambda, which changes no bit of a nonzero sum of finite terms.  A zero lambda (the
// sign of a zero sum) counts as a dependency, and so does a neighbour that is or was not finite: 0 *
// inf has made the sum NaN, and it stays so until the node is updated again.  (Without short circuits:
// the lanes diverged over them; 16 shots of 96 x 96 x 48, per diagonal, adjoint 145.6 -> 138.5 ms.)
PFAST_HD bool adj_depends_exact(double t0, double tn, double vn, double old, double nv) {
    const int en = exponent_of(nv), eo = exponent_of(old);
    return (ordered(t0) > ordered(tn)) | is_zero(vn) | ((en > eo ? en : eo) == 0x7ff);
}

// ------------------------------------------------------------------ 2D
struct ExactGrid2 {
    DivBy x, z;     // dx, dz
    DivBy all;      // 1/dx^2 + 1/dz^2
    int quick, fast;
};

inline ExactGrid2 exact_grid2(double dx, double dz) {
    ExactGrid2 g;
    std::memset(&g, 0, sizeof(g));
    g.quick = dx > 0x1p-20 && dx < 0x1p20 && dz > 0x1p-20 && dz < 0x1p20;
    if (!g.quick) return g;
    g.x = div_by(dx);
    g.z = div_by(dz);
    g.all = div_by(1.0 / dx / dx + 1.0 / dz / dz);
    g.fast = g.x.fast & g.z.fast;
    return g;
}

// The reference's 2D Godunov solution (src/RT_pfsm2d.h:89-102), bit for bit: x-neighbour minimum
// x, z-neighbour minimum z.  The two sums of the reference commute, so nothing is sorted beyond
// the smaller neighbour.  29 FP64 instructions (spacings of few bits) instead of about 95.
template <bool FAST>
PFAST_HD double eik2_exact(double x, double z, double s, const ExactGrid2& g) {
    const bool zlow = bits_of(z) <= bits_of(x);
    const double lo = zlow ? z : x, hi = zlow ? x : z;
    const double dlo = zlow ? g.z.d : g.x.d;
    const double q = lo + dlo * s;
    if (bits_of(q) <= bits_of(hi)) return q;
    double S, C;
    if (in_range(hi) && (is_zero(lo) || in_range(lo)) && slow_in_range(s)) {
        auto dv = [](double v, const DivBy& k) {   // one of the two may be 0 beside the source
            const double r = div_exact<FAST>(v, k);
            return is_zero(v) ? v : r;
        };
        S = dv(dv(x, g.x), g.x) + dv(dv(z, g.z), g.z);
        C = dv(dv(x * x, g.x), g.x) + dv(dv(z * z, g.z), g.z) - s * s;
        const double D = S * S - g.all.d * C;
        return (D >= 0) ? div_exact<false>(S + sqrt_exact(D), g.all) : kUnreached;
    }
    const double A = g.all.d;
    const double B = -2. * (x / g.x.d / g.x.d + z / g.z.d / g.z.d);
    C = x * x / g.x.d / g.x.d + z * z / g.z.d / g.z.d - s * s;
    const double D = B * B - 4 * A * C;
    return (D >= 0) ? (-B + sqrt(D)) / 2. / A : kUnreached;
}

}  // namespace pfast
