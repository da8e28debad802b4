// The plain FP64 updates of exact_arith.h against the reference's expressions, bit for bit (NaN for
// NaN), on arguments far outside those of a survey: slownesses from 0 over the whole exponent range
// to infinity; traveltimes of a caller's field that are NaN, infinite or huge.  Prints "ok <name> <cases>" or "FAIL ..." lines.
#include <algorithm>
#include <cstdio>
#include <random>

#include "exact_arith.h"

using namespace pfast;

static std::mt19937_64 rng(977);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static bool same(double a, double b) { return bits_of(a) == bits_of(b) || (std::isnan(a) && std::isnan(b)); }

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
    {   // neighbour minima of a solve (0 at the source, up to the unreached value, infinite at the grid's faces)
        long long n3 = 0, w3 = 0, n2 = 0, w2 = 0;
        for (int dec = -324; dec <= 310; ++dec)
            for (int i = 0; i < 4000; ++i) {
                double s = std::pow(10.0, dec + uni(0.0, 1.0));   // 0 below the range, infinite above it
                double d[3];
                const double h = spacings[rng() % 11];
                for (double& v : d) v = i % 2 ? spacings[rng() % 11] : h;
                const double base = rng() % 3 ? std::pow(10.0, uni(-9.0, 7.0)) : 0.0;
                double v[3];
                for (double& x : v) {
                    x = std::min(kUnreached, base * (1.0 + uni(0.0, 1.0) * (rng() % 2 ? 1e-3 : 1.0)));
                    const unsigned c = rng() % 24;
                    if (c == 0) x = 0.0;
                    if (c == 1) x = kUnreached;
                    if (c == 2) x = INFINITY;
                }
                const ExactGrid3 g = exact_grid3(d);
                double inv2[3];
                for (int a = 0; a < 3; ++a) inv2[a] = 1.0 / d[a] / d[a];
                const double r = eik3_ref(v[0], v[1], v[2], s, d);
                w3 += !same(r, eik3_exact<false, false>(v[0], v[1], v[2], s, g, inv2));
                if (g.iso) w3 += !same(r, eik3_exact<true, false>(v[0], v[1], v[2], s, g, inv2));
                if (g.iso && g.fast) w3 += !same(r, eik3_exact<true, true>(v[0], v[1], v[2], s, g, inv2));
                ++n3;
                const ExactGrid2 g2 = exact_grid2(d[0], d[1]);
                const double r2 = eik2_ref(v[0], v[1], s, d[0], d[1]);
                w2 += !same(r2, eik2_exact<false>(v[0], v[1], s, g2)) || (g2.fast && !same(r2, eik2_exact<true>(v[0], v[1], s, g2)));
                ++n2;
            }
        report("eik3_slowness", n3, w3);
        report("eik2_slowness", n2, w2);
    }
    {   // adjoint terms of one axis
        const double nan = std::nan("");
        const double Ts[] = {nan, -nan, -(double)INFINITY, -1.7e308, -1e308, -0x1p999, -0x1.fffffffffffffp998, -2e100, -0.4, -0.0, 0.0, 0.3, 9e6};
        const long long inf = bits_of(kUnreached);
        long long n = 0, wrong = 0, taken = 0;
        for (double d : spacings) {
            const DivBy k = div_by(d);
            for (double T0 : Ts) for (double Tp : Ts) for (double Tm : Ts)
                for (int i = 0; i < 40; ++i) {
                    auto L = [&]() -> double {
                        const unsigned c = rng() % 10;
                        return c == 0 ? 0.0 : c == 1 ? -0.0 : c == 2 ? INFINITY : c == 3 ? 1e308 : uni(-3.0, 3.0);
                    };
                    const double Lp = L(), Lm = L();
                    double dr, nr, de, ne;
                    const bool ordinary = adj_ordinary(most_of(most_of(upper_of(T0), upper_of(Tp)), upper_of(Tm)));
                    axis_ref(T0, Tp, Tm, Lp, Lm, d, dr, nr);
                    adj_axis_exact(T0, Tp, Tm, Lp, Lm, k, de, ne);
                    // the others take the expressions as they stand; NaNs without a sign are unreached
                    wrong += ordinary && bits_of(T0) < inf && bits_of(Tp) < inf && bits_of(Tm) < inf &&
                             (!same(dr, de) || !same(nr, ne));
                    taken += ordinary, ++n;
                }
        }
        wrong += taken < n / 8;
        report("adj_axis_any_time", n, wrong);
    }
    {   // marking: a node that does not depend on a neighbour's change keeps every bit under it
        const double vals[] = {0.0, -0.0, INFINITY, -(double)INFINITY, std::nan(""), 1.7e308, 1e300, 1e-310, 1.0, -2.5};
        auto node = [&](double T0, const double* T, const double* L) {
            double den = 0.0, num = 0.0;
            for (int a = 0; a < 3; ++a) {
                double de, ne;
                axis_ref(T0, T[2 * a], T[2 * a + 1], L[2 * a], L[2 * a + 1], 20.0, de, ne);
                den = a ? den + de : de;
                num = a ? num + ne : ne;
            }
            return std::fabs(den) > 1e-9 ? num / den : 0.0;
        };
        long long n = 0, wrong = 0, skipped = 0;
        for (int i = 0; i < 4000000; ++i) {
            const double T0 = uni(0.0, 1.0);
            double T[6], L[6];
            for (double& t : T) t = rng() % 6 ? T0 + uni(-0.1, 0.1) : T0;
            for (double& v : L) v = rng() % 3 ? uni(-30.0, 30.0) : vals[rng() % 10];
            const int c = rng() % 6;
            const double nv = rng() % 2 ? uni(-30.0, 30.0) : vals[rng() % 10], old = L[c];
            const double before = node(T0, T, L);
            L[c] = nv;
            if (!adj_depends_exact(T[c], T0, before, old, nv)) wrong += !same(before, node(T0, T, L)), ++skipped;
            ++n;
        }
        report("adj_marking", n, wrong + (skipped < n / 8));
    }
    {   // marking, 3D forward: the same for a neighbour's change (its axis' other neighbour may hide it),
        // on grids of any spacing and far more steps from the source than a grid has
        long long n = 0, wrong = 0, skipped = 0;
        for (int i = 0; i < 6000000; ++i) {
            double d[3];
            const double h = std::pow(10.0, uni(-3.0, 3.0)), ratio = rng() % 2 ? 1.0 : std::pow(10.0, uni(0.0, 7.0));
            for (double& x : d) x = ratio == 1.0 ? h : h * std::pow(ratio, uni(0.0, 1.0));
            const double s = std::pow(10.0, uni(-5.0, 0.0)), vmax = (1.0 / s) * (rng() % 2 ? 1.0 : uni(1.0, 100.0));
            const int limit = forward_prune_limit(d, vmax);
            const double step = s * *std::min_element(d, d + 3), base = step * std::pow(10.0, rng() % 2 ? uni(0.0, 11.0) : uni(7.0, 9.0));
            double v[3];
            for (double& x : v) {
                const unsigned c = rng() % 8;
                x = c < 3 ? base * (1.0 + std::pow(10.0, uni(-7.0, 0.0))) : c == 3 ? kUnreached : base + step * uni(0.0, 2.0);
            }
            const int a = rng() % 3;
            const double other = rng() % 2 ? kUnreached : v[a] * uni(0.99999, 1.01);
            const double x0 = v[a], x1 = rng() % 2 ? x0 * uni(0.9, 1.1) : x0 + step * uni(-2.0, 2.0);
            v[a] = std::min(x0, other);
            double vn = eik3_ref(v[0], v[1], v[2], s, d);
            if (rng() % 4 == 0) vn *= uni(0.9, 1.0);
            vn = std::min(vn, kUnreached);
            v[a] = std::min(x1, other);
            const double q = eik3_ref(v[0], v[1], v[2], s, d);
            if (x0 >= 0.0 && x1 >= 0.0 && vn >= 0.0 && !forward_depends_exact(forward_change(x0, x1, limit), vn))
                wrong += !same(std::min(vn, q), vn), ++skipped;
            ++n;
        }
        report("fwd_marking", n, wrong + (skipped < n / 50));
        std::printf("%lld of %lld without a dependency\n", skipped, n);
    }
    return bad ? 1 : 0;
}
