// The plain FP64 updates of exact_arith.h against the reference's expressions as they stand, bit
// for bit, on random and edge arguments.  Prints "ok <name> <cases>" or "FAIL ..." lines.
#include <algorithm>
#include <cstdio>
#include <random>

#include "exact_arith.h"

using namespace pfast;

static std::mt19937_64 rng(20240611);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static double any_bits(int emin, int emax) {   // random significand, exponent in [emin, emax]
    const int e = emin + (int)(rng() % (unsigned)(emax - emin + 1));
    return std::ldexp(from_bits((long long)((rng() & 0xfffffffffffffull) | 0x3ff0000000000000ull)), e);
}
static bool same(double a, double b) { return bits_of(a) == bits_of(b); }

static double eik3_ref(double a, double b, double c, double s, const double* d) {
    double da = d[0], db = d[1], dc = d[2], t;
    if (b > a) { t = a; a = b; b = t; t = da; da = db; db = t; }
    if (c > a) { t = a; a = c; c = t; t = da; da = dc; dc = t; }
    if (c > b) { t = b; b = c; c = t; t = db; db = dc; dc = t; }
    double q = dc * s + c;
    if (q <= b) return q;
    double A = dc * dc + db * db, B = -2. * (b * dc * dc + c * db * db);
    double C = dc * dc * b * b + db * db * c * c - db * db * dc * dc * s * s;
    double D = B * B - 4. * A * C;
    q = (D >= 0) ? (-B + std::sqrt(D)) / 2. / A : kUnreached;
    if (q <= a) return q;
    A = 1.0 / da / da + 1.0 / db / db + 1.0 / dc / dc;
    B = -2.0 * (a / da / da + b / db / db + c / dc / dc);
    C = a * a / da / da + b * b / db / db + c * c / dc / dc - s * s;
    D = B * B - 4. * A * C;
    return (D >= 0) ? (-B + std::sqrt(D)) / 2. / A : kUnreached;
}
static double eik2_ref(double a, double b, double s, double dx, double dz) {
    double da = dx, db = dz, t;
    if (b > a) { t = a; a = b; b = t; t = da; da = db; db = t; }
    double q = b + db * s;
    if (q <= a) return q;
    const double A = 1.0 / da / da + 1.0 / db / db, B = -2. * (a / da / da + b / db / db);
    const double C = a * a / da / da + b * b / db / db - s * s, D = B * B - 4 * A * C;
    return (D >= 0) ? (-B + std::sqrt(D)) / 2. / A : kUnreached;
}
static double posr(double x) { return (x + std::fabs(x)) / 2.0; }
static double negr(double x) { return (x - std::fabs(x)) / 2.0; }
static void axis_ref(double T0, double Tp, double Tm, double Lp, double Lm, double d, double& den, double& num) {
    const double gp = -(Tp - T0) / d, gm = -(T0 - Tm) / d;
    den = (posr(gp) - negr(gm)) / d;
    num = (posr(gm) * Lm - negr(gp) * Lp) / d;
}

static int bad = 0;
static void report(const char* name, long long n, long long wrong) {
    std::printf("%s %s %lld\n", wrong ? "FAIL" : "ok", name, wrong ? wrong : n);
    bad += wrong != 0;
}

int main() {
    const double spacings[] = {20.0, 5.0, 12.5, 16.7, 8.3, 0.1, 1.0 / 3.0, 1.0, 4096.0, 3e-6, 7.3e5};
    {   // square root: random values, squares and their neighbours, powers of two, edges of the range
        long long n = 0, wrong = 0;
        for (int i = 0; i < 3000000; ++i) {
            g_seed_error = (float)uni(1.0 - 4e-7, 1.0 + 4e-7);
            double x = any_bits(-110, 110);
            if (i % 4 == 1) { const double m = any_bits(-40, 40); x = m * m; }
            if (i % 4 == 2) x = std::ldexp(1.0, (int)(rng() % 180) - 90);
            if (i % 4 == 3) {   // next to a midpoint of two neighbouring roots
                const double m = any_bits(-40, 40), h = std::ldexp(1.0, std::ilogb(m) - 53);
                x = std::fma(m, m, 2 * m * h);
            }
            if (i % 3 == 1) x = std::nextafter(x, 0.0);
            if (i % 3 == 2) x = std::nextafter(x, 1e300);
            wrong += !same(sqrt_exact(x), std::sqrt(x)), ++n;
        }
        for (double x : {0.0, 0x1p-1074, 0x1p-101, 0x1p100, 1e300, (double)INFINITY}) wrong += !same(sqrt_exact(x), std::sqrt(x)), ++n;
        report("sqrt", n, wrong);
    }
    {   // division by a constant: random values, and values next to multiples and midpoints
        long long n = 0, wrong = 0;
        for (double d : spacings) {
            const DivBy k = div_by(d);
            for (int i = 0; i < 400000; ++i) {
                double x = any_bits(-90, 89);
                if (i % 3 == 1) {   // a quotient next to a 54-bit midpoint, times the divisor
                    const double m = any_bits(-30, 30), h = std::ldexp(1.0, std::ilogb(m) - 53);
                    x = std::fma(m, d, h * d);
                    if (i % 2) x = std::nextafter(x, 0.0);
                } else if (i % 3 == 2) {
                    x = any_bits(-3, 3) * d;
                }
                if (k.fast) wrong += !same(div_exact<true>(x, k), x / d);
                wrong += !same(div_exact<false>(x, k), x / d) || !same(div_mid(-x, k), -x / d) || !same(div_any(-x, k), -x / d);
                const double y = any_bits(-1060, 950);
                wrong += !same(div_any(y, k), y / d) || !same(div_mid(-y, k), -y / d);
                ++n;
            }
            for (double x : {0.0, -0.0, 0x1p-1074, -0x1p-1060, 0x1p-950, 1e300, -1e308, (double)INFINITY})
                wrong += !same(div_any(x, k), x / d) || !same(div_mid(x, k), x / d), ++n;
        }
        report("div", n, wrong);
    }
    for (int mode = 0; mode < 6; ++mode) {   // 3D Godunov update
        long long n = 0, wrong = 0;
        for (int i = 0; i < 1500000; ++i) {
            double d[3];
            const double h = spacings[rng() % 8];
            for (double& v : d) v = mode % 2 ? spacings[rng() % 8] : h;
            double s = 1.0 / uni(1400.0, 6000.0);
            const double step = s * *std::min_element(d, d + 3);
            double base = mode < 2 ? uni(0.0, 3.0) : (mode < 4 ? step * std::exp(uni(0.0, 16.0)) : uni(0.0, 2e4 * step));
            double v[3];
            for (double& x : v) x = base + step * (rng() % 4 ? uni(0.0, 1.2) : uni(0.0, 3.0));
            const unsigned c = rng() % 64;
            if (c == 0) v[rng() % 3] = INFINITY;
            if (c == 1) { v[rng() % 3] = INFINITY; v[rng() % 3] = INFINITY; }
            if (c == 2) v[rng() % 3] = kUnreached;
            if (c == 3) v[0] = v[1] = v[2];
            if (c == 4) v[rng() % 3] = 0.0;
            if (c == 5) for (double& x : v) x = kUnreached;
            if (c == 6) v[rng() % 3] = base;
            if (c == 7) { v[0] = base; v[1] = base; v[2] = base + step / std::sqrt(2.0); }   // at the case boundary
            if (c == 8) { const double f = std::ldexp(1.0, (int)(rng() % 1200) - 600); for (double& x : v) x *= f; s *= f; }
            const ExactGrid3 g = exact_grid3(d);
            double inv2[3];
            for (int a = 0; a < 3; ++a) inv2[a] = 1.0 / d[a] / d[a];
            const double r = eik3_ref(v[0], v[1], v[2], s, d);
            wrong += !same(r, eik3_exact<false, false>(v[0], v[1], v[2], s, g, inv2));
            if (g.iso) wrong += !same(r, eik3_exact<true, false>(v[0], v[1], v[2], s, g, inv2));
            if (g.iso && g.fast) wrong += !same(r, eik3_exact<true, true>(v[0], v[1], v[2], s, g, inv2));
            ++n;
        }
        char name[32];
        std::snprintf(name, sizeof(name), "eik3_%d", mode);
        report(name, n, wrong);
    }
    {   // 2D Godunov update
        long long n = 0, wrong = 0;
        for (int i = 0; i < 3000000; ++i) {
            const double dx = spacings[rng() % 8], dz = rng() % 2 ? dx : spacings[rng() % 8];
            double s = 1.0 / uni(1400.0, 6000.0);
            const double step = s * std::min(dx, dz), base = rng() % 2 ? uni(0.0, 3.0) : step * std::exp(uni(0.0, 14.0));
            double a = base + step * uni(0.0, 1.5), b = base + step * uni(0.0, 1.5);
            const unsigned c = rng() % 32;
            if (c == 0) a = INFINITY;
            if (c == 1) b = kUnreached;
            if (c == 2) a = b;
            if (c == 3) b = 0.0;
            if (c == 4) a = b = kUnreached;
            if (c == 5) { const double f = std::ldexp(1.0, (int)(rng() % 1200) - 600); a *= f; b *= f; s *= f; }
            const ExactGrid2 g = exact_grid2(dx, dz);
            const double r = eik2_ref(a, b, s, dx, dz);
            wrong += !same(r, eik2_exact<false>(a, b, s, g)) || (g.fast && !same(r, eik2_exact<true>(a, b, s, g)));
            ++n;
        }
        report("eik2", n, wrong);
    }
    {   // adjoint terms of one axis
        long long n = 0, wrong = 0;
        for (int i = 0; i < 4000000; ++i) {
            const double d = spacings[rng() % 11];
            const double T0 = uni(0.0, 4.0);
            auto T = [&]() { return rng() % 8 ? T0 + uni(-0.02, 0.02) : (rng() % 2 ? T0 : std::nextafter(T0, 9.0)); };
            auto L = [&]() -> double {
                switch (rng() % 8) {
                    case 0: return 0.0;
                    case 1: return -0.0;
                    case 2: return std::ldexp(uni(-1.0, 1.0), -(int)(rng() % 1080));
                    case 3: return rng() % 64 ? uni(-1e3, 1e3) : (rng() % 2 ? INFINITY : -INFINITY);
                    default: return uni(-30.0, 30.0);
                }
            };
            const double Tp = T(), Tm = T(), Lp = L(), Lm = L();
            double dr, nr, de, ne;
            axis_ref(T0, Tp, Tm, Lp, Lm, d, dr, nr);
            adj_axis_exact(T0, Tp, Tm, Lp, Lm, div_by(d), de, ne);
            const bool nan_both = std::isnan(nr) && std::isnan(ne);
            wrong += !same(dr, de) || (!nan_both && !same(nr, ne));
            ++n;
        }
        report("adj_axis", n, wrong);
    }
    return bad ? 1 : 0;
}
