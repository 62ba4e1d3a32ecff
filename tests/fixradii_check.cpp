// Test harness (CPU): the pair terms of the FP64 form with radii in a finer unit
// than the positions', and the range test of the fixed point
// (cubble_gb300/csrc/fixpair.cuh), against long double arithmetic. Prints one
// line "name value" per quantity. Built and run by tests/test_fixradii.py with
// -ffp-contract=off.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>

#include "../cubble_gb300/csrc/fixpair.cuh"

typedef long double ld;

static ld absl_(ld v) { return v < 0 ? -v : v; }

int main() {
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> U(-1.0, 1.0);
    long inexact = 0, refused = 0, range = 0, count = 0;
    ld force = 0, area = 0;
    const int Bs[] = {58, 55, 50, 44, 41}, Ks[] = {0, 1, 5, 9, 14, 20};
    for (int it = 0; it < 1000000; it++) {
        const int B = Bs[it % 5], K = Ks[it % 6];
        // the largest radius of a foam has 2^60 units at most; down to 2^-8 of it
        const double r1 = std::ldexp(std::exp2(60.0 - 8.0 * std::fabs(U(rng))), -B - K);
        const double r2 = it % 3 ? r1 * std::exp2(-std::fabs(U(rng)))
                                 : std::ldexp(std::exp2(60.0 - 8.0 * std::fabs(U(rng))), -B - K);
        bool far = false;
        const int64_t q1 = cbg::fx_from_double(r1, B + K, far), q2 = cbg::fx_from_double(r2, B + K, far);
        if (far) range++;
        if (ldexpl((ld)q1, -B - K) != (ld)r1 || (std::ldexp(r2, B + K) >= 0x1p52 && ldexpl((ld)q2, -B - K) != (ld)r2)) inexact++;
        const ld x1 = q1, x2 = q2, R = x1 + x2;
        ld v[3] = {U(rng), U(rng), U(rng)};
        const ld len = sqrtl(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) + 1e-9L;
        const ld d = R * (0.3L + 0.7L * std::fabs(U(rng)));
        int64_t e[3];
        for (int a = 0; a < 3; a++) e[a] = (int64_t)(ldexpl(v[a] / len * d, -K));
        const ld x = ldexpl(e[0], K), y = ldexpl(e[1], K), z = ldexpl(e[2], K), m = x * x + y * y + z * z;
        const ld large = std::max(x1, x2);
        if (m > R * R || absl_(m - large * large) < 1e-15L * R * R) continue;
        cbg::FxTerms t;
        if (!cbg::fx_pair<3, true>(e[0], e[1], e[2], q1, q2, B, t, K)) {
            refused++;
            continue;
        }
        count++;
        const ld s = 1 / sqrtl(m) - 1 / R;
        force = std::max(force, std::max(absl_(t.fx - x * s), std::max(absl_(t.fy - y * s), absl_(t.fz - z * s))));
        const ld small = std::min(x1, x2), D = x1 - x2;
        const ld oa = m < large * large ? small * small : (R - sqrtl(m)) * (R + sqrtl(m)) * (m - D * D) / (4 * m);
        area = std::max(area, absl_(ldexpl((ld)t.oa, 2 * (B + K)) - oa) / (R * R));
    }
    // the same integers inside the range, and the range
    long differ = 0;
    for (int it = 0; it < 400000; it++) {
        const int B = it % 7 ? Bs[it % 5] : it % 2 ? 700 : -700;
        const double x = std::ldexp(U(rng), (int)(70 * U(rng)) - B);
        bool far = false;
        const int64_t q = cbg::fx_from_double(x, B, far);
        if (far != (absl_(ldexpl((ld)x, B)) >= 0x1p62L)) range++;
        if (!far && q != cbg::fx_from_double(x, B)) differ++;
    }
    for (double x : {(double)INFINITY, (double)-INFINITY, std::nan(""), 1e300}) {
        bool far = false;
        cbg::fx_from_double(x, 50, far);
        if (!far) range++;
    }
    printf("count %ld\ninexact %ld\nrefused %ld\nrange %ld\ndiffer %ld\n", count, inexact, refused, range, differ);
    printf("force %.3Le\narea %.3Le\n", force, area);
    return 0;
}
