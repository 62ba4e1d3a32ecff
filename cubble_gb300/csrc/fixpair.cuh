// The FP64 form's pair terms in 64-bit fixed point on the integer pipe.
//
// GB300 issues FP64 at 1/64 of its FP32 rate; one FP64 instruction costs the
// issue slots of about 64 others, a 64-bit integer product about ten. The
// predicted positions and radii of the FP64 form are therefore kept as
// integers: positions q = x 2^B (|x| < P, P the power of two that bounds the
// box corners with an eighth to spare, B = 62 - log2 P: never coarser than the
// doubles they come from except below 2^-9 P, where the unit stays 2^-53 of
// P / 2^9), radii in a unit 2^K finer, which the largest radius sets the same
// way (radius_shift: exact down to 2^-8 of it). A bubble beyond either range is
// taken in FP64. Differences are
// then exact, the minimum image an integer compare, and the distance, the
// reciprocals and the products of a pair run in integers normalised to the
// pair's own scale R = r1 + r2:
//   v' = v 2^s with R' in [2^62, 2^63), i.e. R' = 1.x in units of 2^62;
//   squares and products keep their top 64 bits (units 2^-60 of R'^2, against
//   the 2^-53 rounding of every FP64 operation);
//   1/d' and 1/R' start from FP32 estimates and take one third-order step
//   from an exactly computed residual (Householder), to ~2^-55.
// The force d (1/|d| - 1/R) is at most 1 in magnitude and comes out with an
// absolute error of ~2^-54, the chord with ~2^-56 R^2 (as the height of the
// triangle (r1, r2, d), (R^2 - d^2)(d^2 - (r1 - r2)^2) / (4 d^2): no
// cancellation). The results become doubles at the end.
//
// __host__ __device__, so the CPU tests run the same code against extended
// precision.
#pragma once

#include "ff.cuh"

namespace cbg {

#define CB_HD __host__ __device__ __forceinline__
#ifdef __CUDACC__
#define CB_SLOW static __host__ __device__ __noinline__
#else
#define CB_SLOW static __attribute__((noinline))
#endif

CB_HD int fx_clz(uint64_t v) {
    const uint32_t hi = (uint32_t)(v >> 32);
    return hi ? ff_clz(hi) : 32 + ff_clz((uint32_t)v);
}
CB_HD uint64_t fx_mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// x 2^B rounded to nearest, |x| < 2^(63 - B) (beyond: the largest value, with
// the sign of x; NaN too). On the integer pipe, from the bits of x.
CB_HD int64_t fx_from_double(double x, int B) {
    const uint32_t hi = ff_dhi(x), lo = ff_dlo(x);
    const int sh = (int)((hi >> 20) & 0x7ffu) - 1075 + B;  // x = m 2^(sh - B)
    const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
    uint64_t q;
    if (sh >= 0)
        q = sh <= 10 ? m << sh : 0x7fffffffffffffffull;
    else
        q = sh >= -53 ? ((m >> (-sh - 1)) + 1) >> 1 : 0;
    return (hi & 0x80000000u) ? -(int64_t)q : (int64_t)q;
}

// The same for |x| < 2^(62 - B), where differences of two results fit too;
// beyond (NaN too) `far` is set and the result means nothing.
CB_HD int64_t fx_from_double(double x, int B, bool &far) {
    const uint32_t hi = ff_dhi(x), lo = ff_dlo(x);
    const int sh = (int)((hi >> 20) & 0x7ffu) - 1075 + B;
    const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
    far |= sh > 9;
    const uint64_t q = sh >= 0 ? m << (sh & 63) : sh >= -53 ? ((m >> (-sh - 1)) + 1) >> 1 : 0;
    return (hi & 0x80000000u) ? -(int64_t)q : (int64_t)q;
}

// v << s for 0 <= s < 32, in two funnel shifts.
CB_HD uint64_t fx_shl(uint64_t v, int s) {
#ifdef __CUDA_ARCH__
    const uint32_t hi = (uint32_t)(v >> 32), lo = (uint32_t)v;
    return ((uint64_t)__funnelshift_l(lo, hi, s) << 32) | (lo << s);
#else
    return v << s;
#endif
}

// v 2^e2 as a double, rounded to nearest (ties up), v >= 0 and the result in
// the normal range.
CB_SLOW double fx_to_double_small(uint64_t v, int e2, uint32_t sign) {  // v < 2^32
    if (v == 0) return 0.0;
    const int lz = ff_clz((uint32_t)v);  // exact
    const uint64_t b = ((uint64_t)(uint32_t)(1085 - 32 - lz + e2) << 52) + ((v << (lz + 32)) >> 11);
    return ff_mkd((uint32_t)(b >> 32) | sign, (uint32_t)b);
}
CB_HD double fx_to_double(uint64_t v, int e2, uint32_t sign = 0u) {
    const uint32_t h = (uint32_t)(v >> 32);
    if (h == 0u) return fx_to_double_small(v, e2, sign);
    const int lz = ff_clz(h);
    const uint64_t n = fx_shl(v, lz);
    const uint64_t m = (n >> 11) + ((n >> 10) & 1u);  // 53 bits with the hidden one
    const uint64_t b = ((uint64_t)(uint32_t)(1085 - lz + e2) << 52) + m;
    return ff_mkd((uint32_t)(b >> 32) | sign, (uint32_t)b);
}
// The same for values often below 2^32 (no call).
CB_HD double fx_to_double_any(uint64_t v, int e2, uint32_t sign = 0u) {
    if (v == 0) return 0.0;
    const int lz = fx_clz(v);
    const uint64_t n = v << lz;
    const uint64_t m = (n >> 11) + ((n >> 10) & 1u);
    const uint64_t b = ((uint64_t)(uint32_t)(1085 - lz + e2) << 52) + m;
    return ff_mkd((uint32_t)(b >> 32) | sign, (uint32_t)b);
}
CB_HD double fx_to_double_signed(int64_t v, int e2) {
    return v < 0 ? fx_to_double_any((uint64_t)-v, e2, 0x80000000u)
                 : fx_to_double_any((uint64_t)v, e2);
}

// The two halves of v': v' = h 2^32 + 2 l (+ its lowest bit), 0 <= l < 2^31.
struct FxHalves {
    int32_t h, l;
};
CB_HD FxHalves fx_split(int64_t v) {
    return {(int32_t)(v >> 32), (int32_t)((uint32_t)v >> 1)};
}
// v'^2 / 2^64 = h^2 + (h l) / 2^30 to within two units.
CB_HD int64_t fx_square(int64_t v) {
    const FxHalves a = fx_split(v);
    return (int64_t)a.h * a.h + (((int64_t)a.h * a.l) >> 30);
}

CB_HD uint64_t fx_abs(int64_t v) { return (uint64_t)(v < 0 ? -v : v); }

// |(x, y, z)| of integers in units 2^-B: squares normalised to the largest
// component (2^-58), the root in float-float (~2^-46), no FP64 instruction.
template <int DIM>
CB_HD double fx_norm(int64_t x, int64_t y, int64_t z, int B) {
    const uint64_t any = fx_abs(x) | fx_abs(y) | (DIM == 3 ? fx_abs(z) : 0u);
    if (any == 0) return 0.0;
    const int lz = fx_clz(any), s = lz > 2 ? lz - 2 : 0;  // components below 2^62
    uint64_t M = (uint64_t)fx_square(x << s) + (uint64_t)fx_square(y << s);
    if (DIM == 3) M += (uint64_t)fx_square(z << s);  // |v|^2 2^(2 s - 64), in [2^58, 2^62)
    const int t = fx_clz(M) & ~1;  // to [2^62, 2^64): 48 bits keep 2^-47
    M <<= t;
    const float h = (float)(uint32_t)(M >> 40) * 0x1p24f,
                l = (float)(((uint32_t)(M >> 16) & 0xffffffu) + ((uint32_t)(M >> 15) & 1u));
    const double r = ff_to_double(ff_sqrt(fast_two_sum(h, l)));  // sqrt(M) / 2^8
    return ff_mkd(ff_dhi(r) + ((uint32_t)(40 - s - t / 2 - B) << 20), ff_dlo(r));
}

// Two words of a 64-bit integer as FP32 (~2^-24 relative).
CB_HD float fx_float(uint64_t v) {
    return ff_fma((float)(uint32_t)(v >> 32), 4294967296.0f, (float)(uint32_t)v);
}

// 1/sqrt(M 2^-60) in units 2^-58, for 2^54 <= M < 2^62 (values up to 8).
CB_HD uint64_t fx_rsqrt(uint64_t M) {
    const float m = fx_float(M) * 0x1p-60f;
    float y = ff_rsqrt_est(m);
    y = ff_fma(ff_mulr(0.5f, y), ff_fma(-ff_mulr(m, y), y, 1.0f), y);  // Newton: ~2^-24
    const uint32_t Y0 = (uint32_t)(y * 0x1p27f);
    const uint64_t Q = (uint64_t)Y0 * Y0;  // y0^2 2^54
    // e = 1 - m y0^2 in units 2^-61 (|e| < 2^-22), from bits 53... of the product
    const uint64_t W = (fx_mulhi(M, Q) << 11) | ((M * Q) >> 53);
    const int64_t e = (int64_t)((1ull << 61) - W);
    const int32_t E = (int32_t)((e + 128) >> 8);  // units 2^-53
    // y0 (1 + e/2 + 3 e^2 / 8)
    const float ef = (float)E * 0x1p-53f;
    const int32_t c2 = (int32_t)(ff_mulr(ff_mulr(0.375f * ef, ef), y) * 0x1p58f);
    return ((uint64_t)Y0 << 31) + (uint64_t)(((int64_t)(int32_t)Y0 * E) >> 23) + (uint64_t)(int64_t)c2;
}

// 1/(R 2^-62) in units 2^-58, for 2^62 <= R < 2^63 (values in (1/2, 1]).
CB_HD uint64_t fx_rcp(uint64_t R) {
    const float r = fx_float(R) * 0x1p-62f;
    float z = ff_rcp_est(r);
    z = ff_fma(z, ff_fma(-r, z, 1.0f), z);
    const uint32_t Z0 = (uint32_t)(z * 0x1p30f);
    // e = 1 - r z0 in units 2^-60
    const uint64_t W = (uint64_t)(uint32_t)(R >> 32) * Z0 + (((uint64_t)(uint32_t)R * Z0) >> 32);
    const int64_t e = (int64_t)((1ull << 60) - W);
    const int32_t E = (int32_t)((e + 64) >> 7);  // units 2^-53
    const float ef = (float)E * 0x1p-53f;
    const int32_t c2 = (int32_t)(ff_mulr(ff_mulr(ef, ef), z) * 0x1p58f);  // z0 (1 + e + e^2)
    return ((uint64_t)Z0 << 28) + (uint64_t)(((int64_t)(int32_t)Z0 * E) >> 25) + (uint64_t)(int64_t)c2;
}

// The terms of an overlapping pair: the force over f0, d (1/|d| - 1/(r1 + r2))
// (src/kernels.cu:218-233), and the overlap: in 3D the area over pi, in 2D
// the squared half chord, or min(r1, r2)^2 where one centre lies inside the
// other bubble (`inside`; src/kernels.cu:236-256).
struct FxTerms {
    double fx, fy, fz, oa;
    bool inside;
};
// From the exact differences e (minimum image) in units 2^-B and the predicted
// radii q1, q2 in units 2^-(B + K). false where the fixed-point range does not
// hold the pair: centres closer than R/16 ... R/8 (a deeply swallowed bubble),
// a negative predicted radius, or R below 2^(32 + K) units.
template <int DIM, bool GAS>
CB_HD bool fx_pair(int64_t ex, int64_t ey, int64_t ez, int64_t q1, int64_t q2, int B,
                   FxTerms &out, int K = 0) {
    const int64_t R0 = q1 + q2;
    const int s = ff_clz((uint32_t)((uint64_t)R0 >> 32)) - 1, u = s + K;
    if (u > 30 || (q1 | q2) < 0) return false;
    const int64_t R = (int64_t)fx_shl((uint64_t)R0, s);
    const int64_t vx = (int64_t)fx_shl((uint64_t)ex, u), vy = (int64_t)fx_shl((uint64_t)ey, u),
                  vz = DIM == 3 ? (int64_t)fx_shl((uint64_t)ez, u) : 0;
    const FxHalves x = fx_split(vx), y = fx_split(vy), z = fx_split(vz);
    int64_t A = (int64_t)x.h * x.h + (int64_t)y.h * y.h;
    int64_t C = (int64_t)x.h * x.l + (int64_t)y.h * y.l;
    if (DIM == 3) {
        A += (int64_t)z.h * z.h;
        C += (int64_t)z.h * z.l;
    }
    const int64_t M = A + (C >> 30);  // d'^2 2^60
    if (M < (1ll << 54)) return false;
    const uint64_t Y = fx_rsqrt((uint64_t)M);
    const int64_t S0 = (int64_t)(Y - fx_rcp((uint64_t)R));
    const uint64_t S = (uint64_t)(S0 > 0 ? S0 : 0) << 2;  // units 2^-60
    // |e'| 2^62 times s 2^60, top word: units 2^-58
    const uint64_t ax = (uint64_t)(vx < 0 ? -vx : vx), ay = (uint64_t)(vy < 0 ? -vy : vy),
                   az = (uint64_t)(vz < 0 ? -vz : vz);
    out.fx = fx_to_double(fx_mulhi(ax, S), -58, (uint32_t)(ex >> 32) & 0x80000000u);
    out.fy = fx_to_double(fx_mulhi(ay, S), -58, (uint32_t)(ey >> 32) & 0x80000000u);
    out.fz = DIM == 3 ? fx_to_double(fx_mulhi(az, S), -58, (uint32_t)(ez >> 32) & 0x80000000u) : 0.0;
    if (GAS) {
        const int64_t D = (int64_t)fx_shl((uint64_t)(q1 < q2 ? q2 - q1 : q1 - q2), s);
        const int64_t big = (R >> 1) + (D >> 1);  // max(r1, r2)
        const int sc = 62 - u - B;                // R = R' 2^sc
        out.inside = M < fx_square(big);
        uint64_t w;  // units 2^-62
        int e2 = -62 + 2 * sc;
        if (out.inside) {  // min(r1, r2)^2, at its own scale
            const uint64_t q = (uint64_t)((R >> 1) - (D >> 1));
            const int k = ff_clz((uint32_t)(q >> 32)) - 2;  // up to 30
            w = (uint64_t)fx_square((int64_t)fx_shl(q, k)) << 2;
            e2 -= 2 * k;
        } else {
            const int64_t p = fx_square(R) - M, q = M - fx_square(D);
            const uint64_t t = fx_mulhi((uint64_t)(p > 0 ? p : 0), (uint64_t)(q > 0 ? q : 0));
            const uint64_t YY = fx_mulhi(Y << 2, Y << 2);  // y^2 2^56, y <= 2
            w = (fx_mulhi(t, YY) << 12) | ((t * YY) >> 52);  // 4 a^2 2^60
        }
        out.oa = fx_to_double(w, e2);
    }
    return true;
}

#undef CB_HD
#undef CB_SLOW

}  // namespace cbg
