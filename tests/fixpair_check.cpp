// Test harness (CPU): the fixed-point pair terms of the FP64 form
// (cubble_gb300/csrc/fixpair.cuh) against long double arithmetic on the same
// integers. Prints one line "name value" per quantity. Built and run by
// tests/test_fixpair.py with -ffp-contract=off.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "../cubble_gb300/csrc/fixpair.cuh"

typedef long double ld;

static ld absl_(ld v) { return v < 0 ? -v : v; }

struct Worst {
    ld force = 0, area = 0, rms = 0;
    long n = 0, refused = 0, wrong_inside = 0;
};

template <int DIM>
static void one(Worst &w, double dv[3], double r1, double r2, int B) {
    const int64_t q1 = cbg::fx_from_double(r1, B), q2 = cbg::fx_from_double(r2, B);
    int64_t e[3] = {0, 0, 0};
    for (int a = 0; a < DIM; a++) e[a] = cbg::fx_from_double(dv[a], B);
    const ld u = ldexpl(1.0L, -B);
    const ld x = e[0] * u, y = e[1] * u, z = e[2] * u, A = q1 * u, C = q2 * u, R = A + C;
    const ld m = x * x + y * y + z * z;
    if (m > R * R || m == 0) return;
    cbg::FxTerms t;
    if (!cbg::fx_pair<DIM, true>(e[0], e[1], e[2], q1, q2, B, t)) {
        if (m >= 0.14L * 0.14L * R * R) w.refused++;
        return;
    }
    w.n++;
    const ld s = 1.0L / sqrtl(m) - 1.0L / R;
    const ld f[3] = {x * s, y * s, z * s};
    const double g[3] = {t.fx, t.fy, t.fz};
    for (int a = 0; a < DIM; a++) {
        const ld er = absl_(g[a] - f[a]);
        w.force = std::max(w.force, er);
        w.rms += er * er;
    }
    const ld big = std::max(A, C), small = std::min(A, C);
    const bool inside = m < big * big;
    if (inside != t.inside) {  // only within the rounding of the test
        if (absl_(m - big * big) > 1e-17L * R * R) w.wrong_inside++;
        return;
    }
    const ld p = (R - sqrtl(m)) * (R + sqrtl(m)), k = m - (A - C) * (A - C);
    const ld oa = inside ? small * small : p * k / (4 * m);
    w.area = std::max(w.area, absl_(t.oa - oa) / (R * R));
}

int main() {
    std::mt19937_64 rng(2024);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    Worst w3, w2;
    const int Bs[] = {62, 57, 54, 53, 50, 44};
    for (int it = 0; it < 1200000; it++) {
        const int B = Bs[it % 6];
        const double unit = B >= 57 ? 0.05 : 1.0;  // keeps R below 2^(62 - B)
        const double r1 = unit * std::exp2(1.2 * U(rng)), r2 = unit * std::exp2((it % 5 ? 1.2 : 4.0) * U(rng) - (it % 5 ? 0 : 3));
        const double R = r1 + r2;
        double c = std::fabs(U(rng));
        // shallow overlaps, ordinary ones, deep ones, and the containment threshold
        double d = R * (it % 4 == 0 ? 1 - 1e-3 * c * c * c : it % 4 == 1 ? 1 - 0.6 * c : it % 4 == 2 ? std::max(0.14, c) : 1.0);
        if (it % 4 == 3) d = std::max(r1, r2) * (1 + 1e-9 * U(rng));
        double v[3], nn = 0;
        do {
            nn = 0;
            for (double &a : v) nn += (a = U(rng)) * a;
        } while (nn > 1 || nn < 1e-3);
        double v2[3] = {v[0], v[1], 0};
        const double n2 = std::sqrt(v[0] * v[0] + v[1] * v[1] + 1e-300);
        for (double &a : v) a *= d / std::sqrt(nn);
        for (double &a : v2) a *= d / n2;
        if (it % 11 == 0) v[it % 3] = 0.0;  // on an axis plane
        one<3>(w3, v, r1, r2, B);
        one<2>(w2, v2, r1, r2, B);
    }
    printf("force3 %.3Le\nforce2 %.3Le\narea3 %.3Le\narea2 %.3Le\n", w3.force, w2.force, w3.area, w2.area);
    printf("force_rms %.3Le\n", sqrtl(w3.rms / (3 * w3.n)));
    printf("refused %ld\ninside %ld\ncount %ld\n", w3.refused + w2.refused, w3.wrong_inside + w2.wrong_inside, w3.n + w2.n);
    // pairs the range does not hold are refused
    cbg::FxTerms t;
    int taken = 0;
    const int64_t one53 = 1ll << 53;
    taken += cbg::fx_pair<3, true>(one53 / 64, 0, 0, one53, one53, 53, t);  // d = R / 128
    taken += cbg::fx_pair<3, true>(0, 0, 0, one53, one53, 53, t);           // coincident
    taken += cbg::fx_pair<3, true>(one53, 0, 0, 3 * one53, -one53, 53, t);  // a negative radius
    taken += cbg::fx_pair<2, true>(1 << 20, 0, 0, 1 << 20, 1 << 20, 53, t); // below the unit range
    printf("taken_outside %d\n", taken);
    // norms of differences, from one unit to the whole range
    ld worst = 0, mean = 0;
    for (int it = 0; it < 600000; it++) {
        const double span = std::exp2(61.0 - 61.0 * std::fabs(U(rng)));
        int64_t v[3];
        for (int64_t &a : v) a = (int64_t)(U(rng) * span);
        if (it % 5 == 0) v[it % 3] = 0;
        const ld want = sqrtl((ld)v[0] * v[0] + (ld)v[1] * v[1] + (ld)v[2] * v[2]);
        const double got = cbg::fx_norm<3>(v[0], v[1], v[2], 53);
        const ld er = want == 0 ? (got == 0 ? 0 : 1) : (got - ldexpl(want, -53)) / ldexpl(want, -53);
        worst = std::max(worst, absl_(er));
        mean += er;
    }
    printf("norm %.3Le\nnorm_bias %.3Le\n", worst, absl_(mean / 600000));
    // to fixed point and back: the nearest integer, and the same double
    double back = 0, near = 0;
    for (int it = 0; it < 400000; it++) {
        const double x = U(rng) * std::exp2(-12.0 + 20.0 * std::fabs(U(rng)));
        const int64_t q = cbg::fx_from_double(x, 53);
        const double y = cbg::fx_to_double_signed(q, -53);
        near = std::max(near, (double)absl_(ldexpl(x, 53) - q));
        if (std::fabs(x) >= 0.5 && y != x) back += 1;
        if (y != std::ldexp((double)q, -53)) back += 1;
    }
    const double big = 1e300, inf = INFINITY;
    const int64_t top = cbg::fx_from_double(big, 53);
    if (cbg::fx_from_double(-inf, 53) != -top || cbg::fx_from_double(1e-300, 53) != 0) back += 1;
    printf("to_fixed %.3e\nround_trip %.0f\n", near, back);
    return 0;
}
