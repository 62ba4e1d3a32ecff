// One attempt of the Adams-Bashforth-Moulton step, FP64 form:
//   k_predict  : AB2 predict of x, y, (z), r into the packed `pred` rows and
//                the area sums (preIntegrate, src/kernels.cu:40-170)
//   k_pairs    : overlap velocities, pairwise gas flux, overlap areas and
//                flow neighbour sums per pair (pairwiseInteraction,
//                src/kernels.cu:172-337)
//   k_correct  : flow and wall velocities, the mean-field gas exchange, AM2
//                correct, error / expansion / radius maxima, deletion marks,
//                path; its last block takes the accept/reject decision and
//                the dt update of step() (src/simulator.cu:219-246) and, on
//                accept, rotates the buffers and advances the clock as
//                integrate() does (src/simulator.cu:258-334) — on the device
//                (postIntegrate, correct, addFlowVelocity, addWallVelocity,
//                src/kernels.cu:339-593)
// plus the Euler bootstrap of init() (src/simulator.cu:727-787) and the
// energy / volume reductions (src/kernels.cu:941-957, :1013-1024).
#include "common.cuh"

namespace cbg {
namespace {

__device__ __forceinline__ double4_32a ld4(const double *p, int i) {
    return reinterpret_cast<const double4_32a *>(p)[i];
}

// The packed predicted state of bubble i (positions in units 2^-fixb and the
// radius in units 2^-radb, fixpair.cuh; 2D: 1/r beside them): written and read
// back. A bubble that the fixed point does not hold (it lies beyond the range
// after a large dt or as it was loaded, its radius is negative or has outgrown
// what the last search saw, or one of them is NaN) has a marked record, and its
// state in spare rows that only a search uses: its terms are then evaluated in
// FP64 (far_pairs, far_moves and RealPlace below). The loop over the pairs needs
// no test for the mark: it lies 2^62 units from every other bubble (before the
// periodic image), and where that still counts as an overlap its radius, the only
// one below zero, leads to pair_slow, which gives nothing.
constexpr long long kFarRecord = (long long)0x8000000000000000ULL;
__device__ __forceinline__ bool is_far(double4_32a p) {  // |q| < 2^62 in the others
    return __double2hiint(p.x) == (int)0x80000000;
}
struct State {
    double x, y, z, r;
};
template <int DIM>
static __device__ __noinline__ void st_far(double *const *ds, const Ctrl *c, int i, double x,
                                           double y, double z, double r) {
    ds[c->drole[RVQ0]][i] = x;
    ds[c->drole[RVQ1]][i] = y;
    if (DIM == 3) ds[c->drole[RVQ2]][i] = z;
    ds[c->drole[RVQ3]][i] = r;
}
template <int DIM>
__device__ __forceinline__ void st_state(const Bufs &b, const Ctrl *c, int i, double x, double y,
                                         double z, double r, double inv, int fixb, int radb) {
    double4_32a p;
    bool far = __double2hiint(r) < 0;
    double qr = __longlong_as_double(fx_from_double(r, radb, far));
    p.x = __longlong_as_double(fx_from_double(x, fixb, far));
    p.y = __longlong_as_double(fx_from_double(y, fixb, far));
    p.z = DIM == 3 ? __longlong_as_double(fx_from_double(z, fixb, far)) : 0.0;
    if (far) {
        p.x = __longlong_as_double(kFarRecord);
        p.y = p.z = 0.0;
        qr = __longlong_as_double(-1LL);
        b.run->far = 1;
        st_far<DIM>(b.ds, c, i, x, y, z, r);
    }
    (DIM == 3 ? p.w : p.z) = qr;
    if (DIM == 2) p.w = inv;
    reinterpret_cast<double4_32a *>(b.pred)[i] = p;
}
template <int DIM>
__device__ __forceinline__ State ld_state(const double *pred, double *const *ds, const Ctrl *c,
                                          int i, int fixb, int radb) {
    const double4_32a p = ld4(pred, i);
    if (is_far(p))
        return {ds[c->drole[RVQ0]][i], ds[c->drole[RVQ1]][i],
                DIM == 3 ? ds[c->drole[RVQ2]][i] : 0.0, ds[c->drole[RVQ3]][i]};
    auto back = [](double q, int b) { return fx_to_double_signed(__double_as_longlong(q), -b); };
    return {back(p.x, fixb), back(p.y, fixb), DIM == 3 ? back(p.z, fixb) : 0.0,
            back(DIM == 3 ? p.w : p.z, radb)};
}

// ---------------------------------------------------------------- predict
// RES: as a phase of a resident run (common.cuh)
template <int DIM, bool RES = false>
__device__ __forceinline__ void k_predict_body(const Bufs &b, const int vb, const int vg,
                                               RunCtx *rx = nullptr, RunRed *rsm = nullptr) {
    __shared__ double smem[32];
    const Ctrl *c = b.ctrl;
    const int n = c->n;
    const double h = 0.5 * c->dt;
    const int gas = c->use_gas;
    const double *X = drow(b, c, RX), *Y = drow(b, c, RY), *Z = drow(b, c, RZ),
                 *R = drow(b, c, RR);
    const double *V0 = drow(b, c, RV0), *V1 = drow(b, c, RV1), *V2 = drow(b, c, RV2),
                 *V3 = drow(b, c, RV3);
    const double *O0 = drow(b, c, RVO0), *O1 = drow(b, c, RVO1), *O2 = drow(b, c, RVO2),
                 *O3 = drow(b, c, RVO3);
    const int fixb = b.k->fix_b, radb = fixb + c->rad_k;
    double sA = 0.0, sAr = 0.0;
    int na = 0;
    for (int i = first_item<RES>(vb, vg); i < n; i += vg * blockDim.x) {
        // p + 0.5 ts (3 v - vo), src/kernels.cu:48-50
        const double xp = fma(h, fma(3.0, V0[i], -O0[i]), X[i]);
        const double yp = fma(h, fma(3.0, V1[i], -O1[i]), Y[i]);
        double rp = R[i];
        if (gas) rp = fma(h, fma(3.0, V3[i], -O3[i]), rp);
        const double inv = rcp_d(rp);
        const double rsq = rp * rp;
        const double zp = DIM == 3 ? fma(h, fma(3.0, V2[i], -O2[i]), Z[i]) : 0.0;
        if (DIM == 3) reinterpret_cast<double2 *>(b.invr)[i] = make_double2(inv, rsq);
        st_state<DIM>(b, c, i, xp, yp, zp, rp, inv, fixb, radb);
        if (gas) {  // area and area per radius, src/kernels.cu:103-112, with
                    // the constant factor (4 pi, 2 pi) applied to the block sums
            if (DIM == 3) {
                sA += rsq;
                sAr += rp;
            } else {
                sA += rp;
                na++;
            }
        }
    }
    if (DIM == 2) sAr = (double)na;
    constexpr double kArea = DIM == 3 ? 4.0 * kPi : 2.0 * kPi;
    if (RES) {  // the sums are reduced with the pair phase's
        rx->sA = sA;
        rx->sAr = sAr;
        run_barrier(rx);
        return;
    }
    const double tA = kArea * block_reduce(sA, OpSum(), smem);
    const double tAr = kArea * block_reduce(sAr, OpSum(), smem);
    if (threadIdx.x == 0) {
        b.part[0 * vg + vb] = tA;
        b.part[1 * vg + vb] = tAr;
    }
    if (last_block(&b.ctrl->done[DC_PREDICT], vg)) {
        const double fA = fold_partials(b.part + 0 * vg, vg, false, smem);
        const double fAr = fold_partials(b.part + 1 * vg, vg, false, smem);
        if (threadIdx.x == 0) {
            b.ctrl->sumA = fA;
            b.ctrl->sumAr = fAr;
            b.ctrl->done[DC_PREDICT] = 0;
        }
    }
}
CB_KERNEL_PAIR((template <int DIM>), k_predict, (<DIM>), __launch_bounds__(kBlock))


// ------------------------------------------------------------------ pairs
// Overlap velocities, pairwise gas flux and overlap areas
// (pairwiseInteraction, src/kernels.cu:172-337) with FP64 results. GB300
// issues 2 FP64 thread-instructions per SM and cycle and its L1 takes one
// record of a scattered access per cycle, so:
//   * the predicted positions and radii are 64-bit fixed point, and distance,
//     reciprocals, force and overlap of a pair run on the integer pipe, more
//     exactly than in FP64 (fixpair.cuh: force to 9e-17 of f0 at most, FP64
//     4e-16; overlap to 3e-17 R^2, FP64 6e-16). FP64 is left for the gas flux
//     and the sums: 5 instructions per overlapping pair (21 before);
//   * each warp takes 32 consecutive pairs, tests their overlap in FP32 with
//     a guard band (exact integers inside it), and queues the overlapping
//     ones (about 70 % of the listed pairs) in shared memory; the force and
//     gas-exchange arithmetic runs on full warps of overlapping pairs;
//   * the results of 32 pairs are transposed through shared memory and added
//     to the bubbles' rows with FP64 reductions by eight lanes a pair, so
//     that the reductions of one bubble's 64-byte record make one request
//     instead of five (alone: 202 -> 177 us);
//   * overlap areas are accumulated in units of ov_unit (pi in 3D, 2 in 2D);
//     the unit is applied to the global sums and in the correct kernel.
// 3D, N = 10^6, 4.67 10^6 pairs, one GB300: 202 -> 121 us (2D 117 -> 89, 3D
// without gas exchange 141 -> 96). Nothing is saturated now: issue 61 %, L1 61 %
// of its wavefronts, FP64 33 %; three or four blocks per SM make no difference,
// record loads a chunk ahead (108 registers) cost 8 us.
__device__ __forceinline__ void red_add(double *p, double v) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"(v));
}

constexpr int kQueue = 64;  // per-warp queue of overlapping pairs

// Unit of the overlap rows the pair kernels write: pi in 3D (an overlap area
// is pi (chord radius)^2), 2 in 2D (an overlap length is 2 (half chord)).
__host__ __device__ constexpr double ov_unit(int dim) { return dim == 3 ? kPi : 2.0; }

// The end of a pair kernel: the attempt's total overlap area and overlap area
// per radius (src/kernels.cu:264-267; each pair adds 2 A_overlap) from the
// threads' sums sAo and sAor, which are in units of ov_unit, and the
// mean-field factors of every bubble (src/kernels.cu:399-404).
template <int DIM, bool RES>
__device__ __forceinline__ void pairs_fold(const Bufs &b, const int vb, const int vg, double sAo,
                                           double sAor, double *smem, RunCtx *rx, RunRed *rsm) {
    double fAo = 0.0, fAor = 0.0;
    if (RES) {
        const double v[4] = {sAo, sAor, rx->sA, rx->sAr};
        run_reduce<4, 0, 0>(v, nullptr, nullptr, rx->acc->psum, nullptr, nullptr, rsm);
        run_barrier(rx);
        run_clear_other(rx, vb);
        if (threadIdx.x == 0 || threadIdx.x == 32) {  // the two divisions in two warps
            constexpr double kArea = DIM == 3 ? 4.0 * kPi : 2.0 * kPi;
            Ctrl *cc = b.ctrl;
            const double sumA = kArea * __ldcg(&rx->acc->psum[2]);
            if (threadIdx.x == 32) {
                cc->mfb = b.k->kappa * b.k->ain * (double)cc->n / sumA;
            } else {
                const double sumAr = kArea * __ldcg(&rx->acc->psum[3]);
                const double sumAo = (2.0 * ov_unit(DIM)) * __ldcg(&rx->acc->psum[0]);
                const double sumAor = ov_unit(DIM) * __ldcg(&rx->acc->psum[1]);
                cc->mfa = (sumAr - sumAor) / (sumA - sumAo);
                cc->sumA = sumA;
                cc->sumAr = sumAr;
                cc->sumAo = sumAo;
                cc->sumAor = sumAor;
            }
        }
        return;
    } else {
        const double tAo = block_reduce(sAo, OpSum(), smem);
        const double tAor = block_reduce(sAor, OpSum(), smem);
        if (threadIdx.x == 0) {
            b.part[2 * vg + vb] = tAo;
            b.part[3 * vg + vb] = tAor;
        }
        if (!last_block(&b.ctrl->done[DC_PAIRS], vg)) return;
        fAo = fold_partials(b.part + 2 * vg, vg, false, smem);
        fAor = fold_partials(b.part + 3 * vg, vg, false, smem);
    }
    if (threadIdx.x == 0) {
        Ctrl *cc = b.ctrl;
        cc->sumAo = (2.0 * ov_unit(DIM)) * fAo;
        cc->sumAor = ov_unit(DIM) * fAor;
        cc->mfa = (cc->sumAr - cc->sumAor) / (cc->sumA - cc->sumAo);
        cc->mfb = b.k->kappa * b.k->ain * (double)cc->n / cc->sumA;
        cc->done[DC_PAIRS] = 0;
    }
}

// The overlap test for pairs in the FP32 guard band: (r1 + r2)^2 >= d^2 from
// the exact integers (R >= 0 in units 2^-K of the differences'; a unit of
// 2^-60 R^2).
template <int DIM>
static __device__ __noinline__ bool overlap_exact(long long ex, long long ey, long long ez,
                                                  long long R, int K) {
    const long long cut = R >> K;
    if (llabs(ex) > cut || llabs(ey) > cut || (DIM == 3 && llabs(ez) > cut)) return false;
    const int s = fx_clz((unsigned long long)R | 1ull) - 1, u = min(s + K, 63);  // |e| 2^u <= R 2^s
    long long m = fx_square(ex << u) + fx_square(ey << u);
    if (DIM == 3) m += fx_square(ez << u);
    return fx_square(R << s) >= m;
}

// The terms of a pair fx_pair does not take, in FP64: centres much closer than
// the radii, or radii more than 1 : 31 apart (its absolute error of 2^-56 R^2 in
// the overlap is then more than FP64's, which scales with the smaller radius; at
// 1 : 1000 2 10^-12 against 6 10^-15 of it). A radius that its unit does not hold
// exactly is predicted again from the rows. The force goes to rs[0], rs[kT], ...;
// returns the overlap as FxTerms::oa. Nothing for a marked bubble, whose pairs
// far_pairs takes.
// Row length of the transposed results (32 pairs): the 8-byte loads of four
// pairs' components fall on distinct banks, but for the fifth row.
constexpr int kT = 36;
template <int DIM, bool GAS>
static __device__ __noinline__ double pair_slow(long long ex, long long ey, long long ez,
                                                long long q1, long long q2, int K,
                                                const DevConst &k, double *const *ds,
                                                const Ctrl *c, const int2 *ij, double *rs) {
    if ((q1 | q2) < 0) {
#pragma unroll
        for (int t = 0; t < DIM; t++) rs[t * kT] = 0.0;
        return 0.0;
    }
    const double unit = k.fix_unit, runit = ldexp(unit, -K), f0 = k.f0;
    const double dx = (double)ex * unit, dy = (double)ey * unit, dz = (double)ez * unit;
    auto radius = [&](long long q, int i) {
        if (!GAS || q >= (1LL << 52)) return (double)q * runit;
        const double *R = ds[c->drole[RR]], *V = ds[c->drole[RV3]], *O = ds[c->drole[RVO3]];
        return fma(0.5 * c->dt, fma(3.0, V[i], -O[i]), R[i]);  // as k_predict
    };
    const double r1 = radius(q1, ij->x), r2 = radius(q2, ij->y);
    double m = dx * dx;
    m = fma(dy, dy, m);
    if (DIM == 3) m = fma(dz, dz, m);
    const double y = rsqrt_d(m), s = (y - rcp_d(r1 + r2)) * f0;
    rs[0 * kT] = dx * s;
    rs[1 * kT] = dy * s;
    if (DIM == 3) rs[2 * kT] = dz * s;
    // the half chord from the smaller bubble's side: its terms scale with it
    const double lo = fmin(r1, r2), hi = fmax(r1, r2), losq = lo * lo, hisq = hi * hi;
    if (m < hisq) return losq;
    const double w = (losq + (m - hisq)) * y;
    return fabs(fma(-0.25 * w, w, losq));
}

// A listed pair with a member that the fixed point does not hold, in FP64 from
// the states to both bubbles' rows. Returns the overlap (in units of ov_unit)
// and the overlap times the sum of 1/r.
template <int DIM, bool GAS, bool FLOW>
static __device__ __noinline__ double2 pair_far(const double *pred, const double *invr, double *acc,
                                                double *const *ds, const Ctrl *c,
                                                const DevConst *kp, int i, int j) {
    const DevConst &k = *kp;
    const int fixb = k.fix_b, radb = fixb + c->rad_k;
    const State a = ld_state<DIM>(pred, ds, c, i, fixb, radb),
                q = ld_state<DIM>(pred, ds, c, j, fixb, radb);
    double dx = a.x - q.x, dy = a.y - q.y, dz = DIM == 3 ? a.z - q.z : 0.0;
    if (!k.wall[0]) dx = min_image(dx, k.half_iv[0], k.iv[0]);
    if (!k.wall[1]) dy = min_image(dy, k.half_iv[1], k.iv[1]);
    if (DIM == 3 && !k.wall[2]) dz = min_image(dz, k.half_iv[2], k.iv[2]);
    const double m = DIM == 3 ? fma(dz, dz, fma(dy, dy, dx * dx)) : fma(dy, dy, dx * dx);
    const double radii = a.r + q.r;
    if (radii * radii < m) return make_double2(0.0, 0.0);  // NaN: counted in
    const double y = rsqrt_d(m), s = (y - rcp_d(radii)) * k.f0;
    double *ai = acc + (size_t)i * kAcc, *aj = acc + (size_t)j * kAcc;
    const double f[3] = {dx * s, dy * s, dz * s};
#pragma unroll
    for (int t = 0; t < DIM; t++) {
        red_add(ai + t, f[t]);
        red_add(aj + t, neg_bits(f[t]));
    }
    if (FLOW) {
        static constexpr int kV[3] = {RV0, RV1, RV2};
#pragma unroll
        for (int t = 0; t < DIM; t++) red_add(ai + 5 + t, ds[c->drole[kV[t]]][j]);
    }
    if (!GAS) return make_double2(0.0, 0.0);
    const double inv1 = DIM == 3 ? invr[2 * (size_t)i] : pred[4 * (size_t)i + 3];
    const double inv2 = DIM == 3 ? invr[2 * (size_t)j] : pred[4 * (size_t)j + 3];
    const double r1sq = a.r * a.r, r2sq = q.r * q.r;
    double oa;
    if (m < r1sq || m < r2sq) {
        oa = fmin(r1sq, r2sq);
    } else {
        const double w = (r2sq - r1sq + m) * y;
        oa = fabs(fma(-0.25 * w, w, r2sq));
    }
    if (DIM == 2) oa = sqrt(oa);
    const double g = oa * (inv2 - inv1);
    red_add(ai + 3, g);
    red_add(aj + 3, neg_bits(g));
    red_add(ai + 4, oa);
    red_add(aj + 4, oa);
    return make_double2(oa, oa * (inv1 + inv2));
}

// This thread's pairs of that kind, where any bubble is (RunSync::far), in a
// pass of their own and with this thread's share of the sums: the call in the
// loop over all pairs cost an attempt 2 to 3 %.
template <int DIM, bool GAS, bool FLOW, bool RES>
static __device__ __noinline__ double2 far_pairs(const double *pred, const double *invr, double *acc,
                                                 double *const *ds, int *const *ps, const Ctrl *c,
                                                 const DevConst *k, int vb, int vg) {
    double2 sum = make_double2(0.0, 0.0);
    const int np = c->np;
    const int *PI = ps[c->prole[PI0]], *PJ = ps[c->prole[PJ0]];
    for (int p = first_item<RES>(vb, vg); p < np; p += vg * blockDim.x) {
        const int i = PI[p], j = PJ[p];
        if (!is_far(ld4(pred, i)) && !is_far(ld4(pred, j))) continue;
        const double2 t = pair_far<DIM, GAS, FLOW>(pred, invr, acc, ds, c, k, i, j);
        sum.x += t.x;
        sum.y += t.y;
    }
    return sum;
}

// The force times f0 where it is not 1 (a call: inlined, its FP64 products
// are predicated into every pair).
template <int DIM>
static __device__ __noinline__ void scale_force(double f0, double *rs) {
#pragma unroll
    for (int a = 0; a < DIM; a++) rs[a * kT] *= f0;
}

// One radius (in its high words) less than 1/32 of the sum: see pair_slow.
__device__ __forceinline__ bool uneven(long long q1, long long q2) {
    const int a = (int)(q1 >> 32), b = (int)(q2 >> 32);
    return min(a, b) < (a + b) >> 5;
}

// The difference of two fixed-point positions (modulo 2^64: one of them may be
// the mark of a bubble beyond the range).
__device__ __forceinline__ long long fix_diff(double a, double b) {
    return (long long)((unsigned long long)__double_as_longlong(a) -
                       (unsigned long long)__double_as_longlong(b));
}

// A fixed-point length as FP32, in units of 2^32: the signed high word and the
// low one (~2^-24 relative, 2^-24 units where they cancel).
__device__ __forceinline__ float fix_len(long long v) {
    return fmaf((float)(unsigned)v, 0x1p-32f, (float)(int)(v >> 32));
}

template <int DIM, bool GAS, bool FLOW, bool RES = false>
__device__ __forceinline__ void k_pairs_body(const Bufs &b, const int vb, const int vg,
                                             RunCtx *rx = nullptr, RunRed *rsm = nullptr) {
    constexpr int kW = kBlock / 32;
    __shared__ double smem[32];
    // queue slots: the differences, both radii
    constexpr int kR1 = DIM, kSlots = kR1 + 2;
    __shared__ long long qd[kW][kSlots][kQueue];
    __shared__ int2 qij[kW][kQueue];
    // the results of 32 pairs, component by component
    constexpr int kC = GAS ? DIM + 2 : DIM;
    __shared__ double res[kW][kC * kT];
    const Ctrl *c = b.ctrl;
    const DevConst &k = *b.k;
    const int any_far = __ldcg(&b.run->far);
    double sAo = 0.0, sAor = 0.0;
    const int np = c->np;
    const int *PI = b.ps[c->prole[PI0]];
    const int *PJ = b.ps[c->prole[PJ0]];
    const double *V0 = drow(b, c, RV0), *V1 = drow(b, c, RV1), *V2 = drow(b, c, RV2);
    const double f0 = k.f0;
    const bool scaled = __double_as_longlong(f0) != 0x3ff0000000000000LL;
    const int fixb = k.fix_b, radk = c->rad_k;
    const float rscale = __int_as_float((127 - radk) << 23);  // radii in the positions' unit
    const bool px = !k.wall[0], py = !k.wall[1], pz = DIM == 3 && !k.wall[2];
    const long long hx = k.fhq[0], hy = k.fhq[1], hz = k.fhq[2];
    const long long Lx = k.flq[0], Ly = k.flq[1], Lz = k.flq[2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    long long(*Q)[kQueue] = qd[w];
    int2 *QP = qij[w];
    double *RS = res[w];

    // minimum image (wrappedDifference, src/kernels.cu:1094-1114), exact
    auto image = [](long long d, long long half, long long len) {
        if ((unsigned long long)d + half > 2ull * half) d -= d > 0 ? len : -len;
        return d;
    };

    // the force and gas-exchange terms of queued (overlapping) pair e
    // (slot of the ring; its results go to column e)
    auto process = [&](int slot, int e) {
        const int i = QP[slot].x, j = QP[slot].y;
        double inv1 = 0.0, inv2 = 0.0;
        if (GAS) {  // 1/r of k_predict
            inv1 = DIM == 3 ? b.invr[2 * (size_t)i] : b.pred[4 * (size_t)i + 3];
            inv2 = DIM == 3 ? b.invr[2 * (size_t)j] : b.pred[4 * (size_t)j + 3];
        }
        const long long ex = Q[0][slot], ey = Q[1][slot], ez = DIM == 3 ? Q[2][slot] : 0;
        const long long q1 = Q[kR1][slot], q2 = Q[kR1 + 1][slot];
        double oa;
        FxTerms t;
        bool on = true;
        if (!uneven(q1, q2) && fx_pair<DIM, GAS>(ex, ey, ez, q1, q2, fixb, t, radk)) {
            RS[0 * kT + e] = t.fx;
            RS[1 * kT + e] = t.fy;
            if (DIM == 3) RS[2 * kT + e] = t.fz;
            oa = t.oa;
            if (scaled) scale_force<DIM>(f0, RS + e);
        } else {
            oa = pair_slow<DIM, GAS>(ex, ey, ez, q1, q2, radk, k, b.ds, c, QP + slot, RS + e);
            on = (q1 | q2) >= 0;
            if (GAS && !on) inv1 = inv2 = 0.0;
        }
        if (GAS) {  // pairwise gas exchange, src/kernels.cu:236-280; oa in units of ov_unit
            if (DIM == 2) oa = __double_as_longlong(oa) > 0 ? oa * rsqrt_d(oa) : 0.0;
            RS[DIM * kT + e] = oa * (inv2 - inv1);
            RS[(DIM + 1) * kT + e] = oa;
            sAo += oa;
            sAor = fma(oa, inv1 + inv2, sAor);
        }
        if (FLOW && on) {  // src/kernels.cu:298-307 (overlapping pairs only)
            double *ai = b.acc + (size_t)i * kAcc;
            red_add(ai + 5, V0[j]);
            red_add(ai + 6, V1[j]);
            if (DIM == 3) red_add(ai + 7, V2[j]);
        }
    };
    // adds the results of the m queued pairs from `head` on to both bubbles'
    // rows: eight lanes a pair, a component each
    auto scatter = [&](int head, int m) {
        __syncwarp();
        const int q = lane & 7;
        const int slot = DIM == 2 && q >= 2 ? q + 1 : q;  // vx, vy, vz, vr, overlap
#pragma unroll
        for (int e0 = 0; e0 < 32; e0 += 4) {
            const int e = e0 + (lane >> 3);
            if (e < m && q < kC) {
                const double v = RS[q * kT + e];
                const int2 ij = QP[(head + e) & (kQueue - 1)];
                red_add(b.acc + (size_t)ij.x * kAcc + slot, v);
                red_add(b.acc + (size_t)ij.y * kAcc + slot, slot == 4 ? v : neg_bits(v));
            }
        }
        __syncwarp();
    };

    // queued pairs of this warp: cnt of them from `head` on in a ring of kQueue
    int cnt = 0, head = 0;
    const int nch = (np + 31) >> 5;
    const int wb = RES ? blockDim.x >> 5 : kW;  // warps of this block
    int p = ((RES ? w * vg + vb : vb * kW + w) << 5) + lane;
    const int step = (vg * wb) << 5;
    int i1 = 0, j1 = 0;  // the next chunk's pair, loaded a chunk ahead
    if (p < np) {
        i1 = PI[p];
        j1 = PJ[p];
    }
    if (any_far) {  // ahead of the loop: its registers are free
        const double2 t = far_pairs<DIM, GAS, FLOW, RES>(b.pred, b.invr, b.acc, b.ds, b.ps, c, &k,
                                                         vb, vg);
        sAo = t.x;
        sAor = t.y;
    }
    for (; (p >> 5) < nch; p += step) {
        bool over = false;
        const int i = i1, j = j1;
        long long ex = 0, ey = 0, ez = 0, q1 = 0, q2 = 0;
        if (p + step < np) {
            i1 = PI[p + step];
            j1 = PJ[p + step];
        }
        if (FLOW) {
            // i's velocity to j's sum for every pair (src/kernels.cu:191-207),
            // a bubble's components in one request: 3D, N = 3 10^5 64 -> 57 us
            // (2D 35.5 -> 34.7). The overlapping pairs' sums of i, below, are
            // better added one by one: in the free lanes of `scatter` their
            // loads held up its reductions (2D 52.9 -> 58 us per attempt)
            constexpr int kL = DIM == 3 ? 4 : 2;  // lanes a pair, a component each
            const int a = lane & (kL - 1);
            const double *VA = a == 0 ? V0 : a == 1 ? V1 : V2;
#pragma unroll
            for (int e0 = 0; e0 < 32; e0 += 32 / kL) {
                const int e = e0 + lane / kL;
                const int ie = __shfl_sync(0xffffffffu, i, e), je = __shfl_sync(0xffffffffu, j, e);
                if (p - lane + e < np && a < DIM)
                    red_add(b.acc + (size_t)je * kAcc + 5 + a, VA[ie]);
            }
        }
        if (p < np) {
            const double4_32a a = ld4(b.pred, i), q = ld4(b.pred, j);
            q1 = __double_as_longlong(DIM == 3 ? a.w : a.z);
            q2 = __double_as_longlong(DIM == 3 ? q.w : q.z);
            ex = fix_diff(a.x, q.x);
            ey = fix_diff(a.y, q.y);
            if (px) ex = image(ex, hx, Lx);
            if (py) ey = image(ey, hy, Ly);
            if (DIM == 3) {
                ez = fix_diff(a.z, q.z);
                if (pz) ez = image(ez, hz, Lz);
            }
            // overlap test (r1 + r2)^2 >= d^2: in FP32 outside a 1e-5 guard
            // band (the differences exact, ~2^-22 relative as FP32), else on
            // the integers
            const float fx = fix_len(ex), fy = fix_len(ey), fz = DIM == 3 ? fix_len(ez) : 0.f;
            float m32 = fx * fx;
            m32 = fmaf(fy, fy, m32);
            if (DIM == 3) m32 = fmaf(fz, fz, m32);
            const long long R = q1 + q2;
            const float R32 = fix_len(R) * rscale;
            const float RR = R32 * R32;
            if (m32 < RR * (1.f - 1e-5f))
                over = true;
            else if (!(m32 > RR * (1.f + 1e-5f)))
                over = overlap_exact<DIM>(ex, ey, ez, max(R, 0LL), radk);
        }
        const unsigned mask = __ballot_sync(0xffffffffu, over);
        if (over) {
            const int e = (head + cnt + __popc(mask & below)) & (kQueue - 1);
            QP[e] = make_int2(i, j);
            Q[0][e] = ex;
            Q[1][e] = ey;
            if (DIM == 3) Q[2][e] = ez;
            Q[kR1][e] = q1;
            Q[kR1 + 1][e] = q2;
        }
        cnt += __popc(mask);
        __syncwarp();
        if (cnt >= 32) {  // a full warp of overlapping pairs
            process((head + lane) & (kQueue - 1), lane);
            scatter(head, 32);
            head = (head + 32) & (kQueue - 1);
            cnt -= 32;
        }
    }
    if (lane < cnt) process((head + lane) & (kQueue - 1), lane);
    scatter(head, cnt);
    pairs_fold<DIM, RES>(b, vb, vg, sAo, sAor, smem, rx, rsm);
}
CB_KERNEL_PAIR((template <int DIM, bool GAS, bool FLOW>), k_pairs, (<DIM, GAS, FLOW>), __launch_bounds__(kBlock, 4))


// ---------------------------------------------------------------- correct
// |a - b| of fixed-point positions (any two of them)
__device__ __forceinline__ unsigned long long fix_gap(long long a, long long b) {
    const unsigned long long ua = (unsigned long long)a, ub = (unsigned long long)b;
    return a > b ? ua - ub : ub - ua;
}

// The velocity of a bubble that touches a wall (touchesWall,
// src/kernels.cu:553-566): d from the wall, which lies below or above it.
static __device__ __noinline__ double wall_velocity(double f0, double r, double d, bool below) {
    const double v = f0 * (1.0 - d / r);
    return below ? v : -v;
}

// A predicted position against the flow's box and the walls: as fixed point
// (exact comparisons), and in FP64 for a bubble the fixed point does not hold.
struct FixPlace {
    long long q[3];
    long long r;  // in units 2^-(fix_b + rad_k)
    int rad_k;
    // in the positions' unit, rounded down: a distance d <= r where d <= rad
    __device__ __forceinline__ unsigned long long rad() const { return fx_abs(r) >> rad_k; }
    // addFlowVelocity, src/kernels.cu:497-544: between the faces or touching one
    __device__ __forceinline__ bool in_flow(const DevConst &k, int a) const {
        return (q[a] < k.vhq[a] && q[a] > k.vlq[a]) || fix_gap(k.vlq[a], q[a]) <= rad() ||
               fix_gap(k.vhq[a], q[a]) <= rad();
    }
    // touches the nearer wall, the upper one of two
    __device__ __forceinline__ bool touches(const DevConst &k, int a, double &velocity) const {
        const unsigned long long dl = fix_gap(q[a], k.wlq[a]), dh = fix_gap(q[a], k.whq[a]);
        const bool low = dl < dh;
        const unsigned long long d = low ? dl : dh;
        if (d > rad()) return false;
        velocity = wall_velocity(k.f0, fx_to_double_signed(r, -k.fix_b - rad_k),
                                 fx_to_double_any(d, -k.fix_b),
                                 q[a] >= (low ? k.wlq[a] : k.whq[a]));
        return true;
    }
    __device__ __forceinline__ double at(const DevConst &k, int a) const {
        return fx_to_double_signed(q[a], -k.fix_b);
    }
};
struct RealPlace {
    double x[3], r;
    __device__ __forceinline__ bool in_flow(const DevConst &k, int a) const {
        const double lo = k.flow_lbb[a] - x[a], hi = k.flow_tfr[a] - x[a];
        return (hi > 0.0 && lo < 0.0) || lo * lo <= r * r || hi * hi <= r * r;
    }
    __device__ __forceinline__ bool touches(const DevConst &k, int a, double &velocity) const {
        const double lo = x[a] - k.lbb[a], hi = x[a] - k.tfr[a];
        const double d = lo * lo < hi * hi ? lo : hi;
        if (!(r * r >= d * d)) return false;
        velocity = wall_velocity(k.f0, r, fabs(d), !(d < 0.0));
        return true;
    }
    __device__ __forceinline__ double at(const DevConst &, int a) const { return x[a]; }
};

// 1 / (a number of neighbours), 0 for none (src/kernels.cu:500-502)
constexpr int kInvCounts = 32;
static __device__ const double kInvCount[kInvCounts] = {
    0.0,      1.0 / 1,  1.0 / 2,  1.0 / 3,  1.0 / 4,  1.0 / 5,  1.0 / 6,  1.0 / 7,
    1.0 / 8,  1.0 / 9,  1.0 / 10, 1.0 / 11, 1.0 / 12, 1.0 / 13, 1.0 / 14, 1.0 / 15,
    1.0 / 16, 1.0 / 17, 1.0 / 18, 1.0 / 19, 1.0 / 20, 1.0 / 21, 1.0 / 22, 1.0 / 23,
    1.0 / 24, 1.0 / 25, 1.0 / 26, 1.0 / 27, 1.0 / 28, 1.0 / 29, 1.0 / 30, 1.0 / 31};
static __device__ __noinline__ double inv_count(int n) { return n > 0 ? 1.0 / (double)n : 0.0; }

// Flow, shear and wall terms of the velocity (addFlowVelocity,
// addWallVelocity, src/kernels.cu:497-593) as a call taken only when one of
// them is on: inlined, their FP64 arithmetic would be predicated into every
// bubble's path and take FP64 issue slots. The tests of the flow's box and of
// the walls are comparisons of the fixed-point positions (exact), 1/neighbours
// comes from a table and only bubbles that touch a wall divide: two or three
// FP64 instructions instead of ~55 for a bubble in a flow between walls.
struct Vel3 {
    double x, y, z;
};
template <int DIM, typename Place>
static __device__ __noinline__ Vel3 boundary_velocity(const DevConst &k, int flow, int shear,
                                                      double drag, double vpx, double vpy,
                                                      double vpz, Place at, double f0, double f1,
                                                      double f2, int nn) {
    if (flow) {  // addFlowVelocity, src/kernels.cu:497-544
        if (at.in_flow(k, 0) && at.in_flow(k, 1) && (DIM == 2 || at.in_flow(k, 2))) {
            vpx += k.flow_vel[0];
            vpy += k.flow_vel[1];
            if (DIM == 3) vpz += k.flow_vel[2];
        } else {
            const double inv = (unsigned)nn < (unsigned)kInvCounts ? kInvCount[nn] : inv_count(nn);
            vpx = fma(inv, f0, vpx);
            vpy = fma(inv, f1, vpy);
            if (DIM == 3) vpz = fma(inv, f2, vpz);
        }
    }
    if (shear)  // linear shear along x over the last axis (cb_config.shear_speed)
        vpx += k.shear * ((at.at(k, DIM - 1) - k.lbb[DIM - 1]) * k.shear_il - 1.0);
    if (k.any_wall) {  // addWallVelocity, src/kernels.cu:546-593
        double xDrag = 1.0, yDrag = 1.0, velocity = 0.0;
        if (k.wall[0] && at.touches(k, 0, velocity)) {
            vpx += velocity;
            vpy *= drag;
            vpz *= drag;
            xDrag = drag;
        }
        if (k.wall[1] && at.touches(k, 1, velocity)) {
            vpx *= drag;
            vpy += velocity * xDrag;
            vpz *= drag;
            yDrag = drag;
        }
        if (k.wall[2] && at.touches(k, 2, velocity)) {
            vpx *= drag;
            vpy *= drag;
            vpz += velocity * xDrag * yDrag;
        }
    }
    return {vpx, vpy, vpz};
}

// The step error of a bubble, its distance from where the last search saw it
// and its path increment, in FP64: for one of whose positions the fixed point
// does not hold.
struct Moves {
    double err, dist, inc;
};
static __device__ __forceinline__ double norm3(double x, double y, double z) {
    const double s = fma(z, z, fma(y, y, x * x));
    return s > 0.0 ? sqrt(s) : 0.0;
}
template <int DIM>
static __device__ __noinline__ Moves far_moves(const double *pred, double *const *ds, const Ctrl *c,
                                               int i, int fixb, double cx, double cy, double cz,
                                               double cr) {
    auto row = [&](int role) { return ds[c->drole[role]][i]; };
    const State p = ld_state<DIM>(pred, ds, c, i, fixb, fixb + c->rad_k);
    Moves m;
    long long e = 0;  // a NaN counts as the largest error
    e = max_bits(e, abs_bits(p.x - cx));
    e = max_bits(e, abs_bits(p.y - cy));
    if (DIM == 3) e = max_bits(e, abs_bits(p.z - cz));
    if (c->use_gas) e = max_bits(e, abs_bits(p.r - cr));
    m.err = __longlong_as_double(e);
    m.dist = norm3(cx - row(RS0), cy - row(RS1), DIM == 3 ? cz - row(RS2) : 0.0);
    if (c->use_gas) m.dist += cr - row(RS3);
    m.inc = norm3(row(RX) - cx, row(RY) - cy, DIM == 3 ? row(RZ) - cz : 0.0);
    return m;
}

// FP64 issue and latency bound in its first forms (46 FP64 instructions a
// bubble, 105 us at 3D, N = 10^6). The predictor-corrector error, the
// expansion since the last search and the path increment are differences of
// nearby positions: they are taken in the fixed point of the prediction
// (exact; the corrected and saved positions are converted on the integer
// pipe), which leaves the updates, the gas exchange and the volume to FP64:
// 105 -> 92 us; with the row pointers in shared memory and every load ahead
// of the first store 85 us (2D 105 -> 74). Three blocks per SM; two: 2D 82 us,
// four: 90 us (200 bytes of spills).
// x / 2 for x > 0 well inside the range, on the exponent.
__device__ __forceinline__ double half_of(double x) {
    return __hiloint2double(__double2hiint(x) - (1 << 20), __double2loint(x));
}
// 4 x for x > 0 well inside the range, on the exponent.
__device__ __forceinline__ double times4(double x) {
    return __hiloint2double(__double2hiint(x) + (2 << 20), __double2loint(x));
}

template <int DIM, bool RES = false>
__device__ __forceinline__ void k_correct_body(const Bufs &b, const int vb, const int vg,
                                               RunCtx *rx = nullptr, RunRed *rsm = nullptr) {
    __shared__ double smem[32];
    __shared__ int ismem[32];
    Ctrl *c = b.ctrl;
    const DevConst &k = *b.k;
    const int n = c->n;
    const double ts = c->dt;
    const double h = 0.5 * ts;
    const int gas = c->use_gas, path = c->inc_path;
    const int flow = c->use_flow && !k.shear_on, shear = c->use_flow && k.shear_on;
    // row pointers from a table in shared memory (tab_ptr, common.cuh; a
    // resident run has its tables there already): 128 -> 80 registers
    __shared__ unsigned long long tab[RES ? 1 : ND_ROLES];
    if (!RES) {
        if (threadIdx.x < ND_ROLES)
            tab[threadIdx.x] = reinterpret_cast<unsigned long long>(b.ds[c->drole[threadIdx.x]]);
        __syncthreads();
    }
#define CB_D(r) (RES ? drow(b, c, r) : reinterpret_cast<double *>(tab_ptr(tab, r)))
    const int *NN = irow(b, c, INN);
    // mean-field factors, src/kernels.cu:399-408 (uniform over bubbles).
    // The overlap row ov and the pairwise rate are in units of ov_unit, and
    // so is the area here: 4 r^2 (3D), pi r (2D); the unit goes into kq, the
    // factor K ov_unit / area = kq / r^2 (/ r)
    const double mfa = c->mfa, mfb = c->mfb;
    const double kq = DIM == 3 ? k.K * 0.25 : k.K * (1.0 / kPi);
    const double drag = 1.0 - k.wall_drag;
    const int fixb = k.fix_b, radk = c->rad_k;
    long long merr = 0, mrad = 0, mexp = 0;
    double vol = 0.0;
    const int marks = c->marks;
    int ndel = 0, bad = 0;
    for (int i = first_item<RES>(vb, vg); i < n; i += vg * blockDim.x) {
        double *acc = b.acc + (size_t)i * kAcc;
        const double4_32a a0 = reinterpret_cast<const double4_32a *>(acc)[0];
        double4_32a a1;
        a1.x = a1.y = a1.z = a1.w = 0.0;
        if (gas || flow) a1 = reinterpret_cast<const double4_32a *>(acc)[1];
        double vpx = a0.x, vpy = a0.y, vpz = a0.z, vpr = a0.w;
        const double ov = a1.x;
        const double4_32a p = ld4(b.pred, i);
        // every input up front (a load cannot move across a store the
        // compiler thinks may alias it)
        const double err0 = CB_D(RERR)[i], path0 = path ? CB_D(RPATH)[i] : 0.0;
        const double x0 = CB_D(RX)[i], y0 = CB_D(RY)[i], z0 = DIM == 3 ? CB_D(RZ)[i] : 0.0;
        const double s0 = CB_D(RS0)[i], s1 = CB_D(RS1)[i], s2 = DIM == 3 ? CB_D(RS2)[i] : 0.0;
        const double v0 = CB_D(RV0)[i], v1 = CB_D(RV1)[i], v2 = DIM == 3 ? CB_D(RV2)[i] : 0.0;
        double v3 = 0.0, r0 = 0.0, s3 = 0.0;
        double2 ri = make_double2(0.0, 0.0);  // (1/rp, rp^2) of k_predict
        if (gas) {
            v3 = CB_D(RV3)[i];
            r0 = CB_D(RR)[i];
            s3 = CB_D(RS3)[i];
            if (DIM == 3) ri = reinterpret_cast<const double2 *>(b.invr)[i];
        }
        const long long qx = __double_as_longlong(p.x), qy = __double_as_longlong(p.y),
                        qz = DIM == 3 ? __double_as_longlong(p.z) : 0,
                        qr = __double_as_longlong(DIM == 3 ? p.w : p.z);
        bool far = is_far(p);
        if (flow | shear | k.any_wall) {
            const int nn = flow ? NN[i] : 0;
            Vel3 v;
            if (far) {
                const State f = ld_state<DIM>(b.pred, b.ds, c, i, fixb, fixb + radk);
                v = boundary_velocity<DIM>(k, flow, shear, drag, vpx, vpy, vpz,
                                           RealPlace{{f.x, f.y, f.z}, f.r}, a1.y, a1.z, a1.w, nn);
            } else {
                v = boundary_velocity<DIM>(k, flow, shear, drag, vpx, vpy, vpz,
                                           FixPlace{{qx, qy, qz}, qr, radk}, a1.y, a1.z, a1.w, nn);
            }
            vpx = v.x;
            vpy = v.y;
            vpz = v.z;
        }
        // AM2 correct x + 0.5 ts (v + vp), src/kernels.cu:487-495 and :366-387
        const double cx = fma(h, v0 + vpx, x0);
        const double cy = fma(h, v1 + vpy, y0);
        const long long fx = fx_from_double(cx, fixb, far), fy = fx_from_double(cy, fixb, far);
        // the largest |predicted - corrected|, in units 2^-fixb
        uint64_t em = max(fx_abs(qx - fx), fx_abs(qy - fy));
        double cz = 0.0;
        long long fz = 0, sz = 0;
        if (DIM == 3) {
            cz = fma(h, v2 + vpz, z0);
            fz = fx_from_double(cz, fixb, far);
            em = max(em, fx_abs(qz - fz));
            sz = fz - fx_from_double(s2, fixb, far);
        }
        // distance from the position of the last search; only its maximum
        // over the foam is used (the search trigger)
        double dist = fx_norm<DIM>(fx - fx_from_double(s0, fixb, far),
                                   fy - fx_from_double(s1, fixb, far), sz, fixb);
        far |= em >> (63 - radk) != 0;
        em <<= radk;  // in the radius's unit
        int del = 0;
        double cr = 0.0;
        if (gas) {  // mean-field gas exchange and radius, src/kernels.cu:390-431
            double inv, area;
            if (DIM == 3) {
                inv = ri.x;
                area = times4(ri.y);
            } else {
                inv = p.w;
                // too small for its unit (or marked): predicted again
                area = kPi * (qr >= (1LL << 52) ? fx_to_double((uint64_t)qr, -(fixb + radk))
                                                : fma(h, fma(3.0, v3, -CB_D(RVO3)[i]), r0));
            }
            double vr = mfa - inv;
            vr *= mfb * (area - ov);
            vr += vpr;
            vr *= DIM == 3 ? kq * (inv * inv) : kq * inv;
            vpr = vr;
            cr = fma(h, v3 + vr, r0);
            em = max(em, fx_abs(qr - fx_from_double(cr, fixb + radk, far)));
            dist += cr - s3;
            if (__double_as_longlong(cr) > __double_as_longlong(k.min_rad)) {  // cr > minRad
                vol = fma(DIM == 3 ? cr * cr : cr, cr, vol);
            } else {
                del = 1;
                ndel++;
            }
            mrad = max_bits(mrad, cr);
            CB_D(RRN)[i] = cr;
            CB_D(RVP3)[i] = vpr;
            bad |= !finite_bits(cr);
        }
        if (del | marks) b.delflag[i] = del;
        double inc = 0.0;
        if (path)  // src/kernels.cu:437-451; the increment to ~2^-46
            inc = fx_norm<DIM>(fx_from_double(x0, fixb, far) - fx,
                               fx_from_double(y0, fixb, far) - fy,
                               DIM == 3 ? fx_from_double(z0, fixb, far) - fz : 0, fixb);
        long long e = __double_as_longlong(fx_to_double_any(em, -(fixb + radk)));
        if (far) {
            const Moves m = far_moves<DIM>(b.pred, b.ds, c, i, fixb, cx, cy, cz, cr);
            e = __double_as_longlong(m.err);
            dist = m.dist;
            inc = m.inc;
        }
        mexp = max_bits(mexp, dist);
        if (path) CB_D(RPATHN)[i] = path0 + inc;
        CB_D(RERR)[i] = __longlong_as_double(max(e, __double_as_longlong(err0)));  // both >= 0
        merr = max(merr, e);
        CB_D(RXN)[i] = cx;
        CB_D(RYN)[i] = cy;
        CB_D(RVP0)[i] = vpx;
        CB_D(RVP1)[i] = vpy;
        if (DIM == 3) {
            CB_D(RZN)[i] = cz;
            CB_D(RVP2)[i] = vpz;
        }
        bad |= !(finite_bits(cx) && finite_bits(cy) && finite_bits(cz));
        if (b.dbg_ov) b.dbg_ov[i] = ov_unit(DIM) * ov;
        // leave the accumulators zeroed for the next attempt
        double4_32a zero;
        zero.x = zero.y = zero.z = zero.w = 0.0;
        reinterpret_cast<double4_32a *>(acc)[0] = zero;
        if (gas || flow) reinterpret_cast<double4_32a *>(acc)[1] = zero;
    }
#undef CB_D
    if (RES) {
        const long long m[3] = {merr, mrad, mexp};
        const int cn[2] = {ndel, bad};
        run_reduce<1, 3, 2>(&vol, m, cn, rx->acc->csum, rx->acc->cmax, rx->acc->cnt, rsm);
        run_barrier(rx);
        run_finish<DIM>(c, k, rx->acc, ts, rx->leave, [] {});
        return;
    }
    long long *lsm = reinterpret_cast<long long *>(smem);
    const double tErr = __longlong_as_double(block_max_bits(merr, lsm));
    const double tRad = __longlong_as_double(block_max_bits(mrad, lsm));
    const double tExp = __longlong_as_double(block_max_bits(mexp, lsm));
    const double tVol = block_reduce(vol, OpSum(), smem);
    const int tDel = block_reduce_int(ndel, ismem);
    const int tBad = block_reduce_int(bad, ismem);
    const int G = vg;
    if (threadIdx.x == 0) {
        b.part[0 * G + vb] = tErr;
        b.part[1 * G + vb] = tRad;
        b.part[2 * G + vb] = tExp;
        b.part[3 * G + vb] = tVol;
        b.part[4 * G + vb] = (double)tDel;
        b.part[5 * G + vb] = (double)tBad;
    }
    if (!last_block(&c->done[DC_CORRECT], vg)) return;
    const double fErr = fold_partials(b.part + 0 * G, G, true, smem);
    const double fRad = fold_partials(b.part + 1 * G, G, true, smem);
    const double fExp = fold_partials(b.part + 2 * G, G, true, smem);
    const double fVol = fold_partials(b.part + 3 * G, G, false, smem);
    const double fDel = fold_partials(b.part + 4 * G, G, false, smem);
    const double fBad = fold_partials(b.part + 5 * G, G, false, smem);
    if (threadIdx.x != 0) return;
    b.run->far = 0;
    finish_attempt<DIM>(c, k, {fErr, fRad, fExp, fVol, (int)fDel, (int)fBad});
}
CB_KERNEL_PAIR((template <int DIM>), k_correct, (<DIM>), __launch_bounds__(kBlock, 3))


// ----------------------------------------------------------- resident run
// Attempts of a foam inside one cooperative launch (see common.cuh; where it
// is taken and what it measured: kRunCapacity, context.cu). BPS blocks per SM:
// two (128 registers) have the lower latency, three (80, some spills) the
// higher throughput.
template <int DIM, bool GAS, bool FLOW, int BPS>
__global__ void __launch_bounds__(kBlock, BPS) k_run(Bufs b, const Bufs *foams,
                                                    const RunBlock *map, RunRound *round, Ctrl *mirror,
                                                    long long n_steps) {
    __shared__ RunShared rs;
    __shared__ RunRed rsm;
    int vb = blockIdx.x, vg = gridDim.x;
    if (map) {  // batched: every foam its own blocks, barrier and loop
        const RunBlock w = map[blockIdx.x];
        b = foams[w.foam];
        vb = w.vb;
        vg = w.vg;
        if (!(b.ctrl->bsel & SEL_ATTEMPT)) return;
    }
    Ctrl *ctrl = b.ctrl;
    RunCtx rx{b.run, nullptr, 0u, (unsigned)vg, &rs.failed, 0.0, 0.0, nullptr};
    run_enter(&rs, b, n_steps);
    if (round) rx.leave = &rs.leave;
    RunWait wait;
    int attempts = 0;
    while (run_more(&rs, attempts)) {
        run_begin(&rx, attempts);
        k_predict_body<DIM, true>(b, vb, vg, &rx, &rsm);
        __syncthreads();
        run_wait_look(&wait, round, vb);
        k_pairs_body<DIM, GAS, FLOW, true>(b, vb, vg, &rx, &rsm);
        __syncthreads();
        run_wait_add(&wait, round, vb, rx.acc);
        k_correct_body<DIM, true>(b, vb, vg, &rx, &rsm);
        attempts++;
    }
    run_exit(&rs, ctrl, mirror, &rx, vb, round, attempts);
}

// --------------------------------------------------------------- bootstrap
// phase 0: pred := (x, r), vo := 0, path := 0
// phase 1: euler pred += acc * dt (src/kernels.cu:959-969), acc := 0
// phase 2: vo := acc (= F(x + dt F(x))), acc := 0
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_boot(Bufs b, int phase) {
    const Ctrl *c = b.ctrl;
    const int n = c->n;
    const double ts = c->dt;
    const double *X = drow(b, c, RX), *Y = drow(b, c, RY), *Z = drow(b, c, RZ),
                 *R = drow(b, c, RR);
    double *O0 = drow(b, c, RVO0), *O1 = drow(b, c, RVO1), *O2 = drow(b, c, RVO2),
           *O3 = drow(b, c, RVO3), *PATH = drow(b, c, RPATH);
    const int fixb = b.k->fix_b, radb = fixb + c->rad_k;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double *acc = b.acc + (size_t)i * kAcc;
        if (phase == 0) {
            const double r = R[i];
            const double inv = 1.0 / r, rsq = r * r;
            if (DIM == 3) reinterpret_cast<double2 *>(b.invr)[i] = make_double2(inv, rsq);
            st_state<DIM>(b, c, i, X[i], Y[i], DIM == 3 ? Z[i] : 0.0, r, inv, fixb, radb);
            O0[i] = O1[i] = O2[i] = O3[i] = 0.0;
            PATH[i] = 0.0;
        } else {
            double4_32a a = reinterpret_cast<double4_32a *>(acc)[0];
            if (phase == 1) {
                const State p = ld_state<DIM>(b.pred, b.ds, c, i, fixb, radb);
                st_state<DIM>(b, c, i, p.x + a.x * ts, p.y + a.y * ts, p.z + a.z * ts, p.r,
                              b.pred[4 * (size_t)i + 3], fixb, radb);
            } else {
                O0[i] = a.x;
                O1[i] = a.y;
                if (DIM == 3) O2[i] = a.z;
            }
            a.x = a.y = a.z = a.w = 0.0;
            reinterpret_cast<double4_32a *>(acc)[0] = a;
        }
    }
}

// ------------------------------------------------------- energy, volume
// sqrt(m) to half an ulp or so with 5 FP64 instructions: m / sqrt(m) and one
// correction from its residual.
static __device__ __noinline__ double sqrt_far(double m) { return sqrt(m); }
__device__ __forceinline__ double sqrt_d(double m) {
    if (!ff_in_range(m)) return sqrt_far(m);
    const double y = rsqrt_d_core(m), s = m * y;
    return fma(fma(-s, s, m), half_of(y), s);
}

// potentialEnergy, src/kernels.cu:941-957, on the current positions. FP64
// bound: with the IEEE square root, an FP64 minimum image and no test for
// pairs well apart a call took 347 us at 3D, N = 10^6 (2D 153), now 168 (87).
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_energy(Bufs b, int per_bubble) {
    __shared__ double smem[32];
    Ctrl *c = b.ctrl;
    const DevConst &k = *b.k;
    const int np = c->np;
    const int *PI = b.ps[c->prole[PI0]];
    const int *PJ = b.ps[c->prole[PJ0]];
    const double *X = drow(b, c, RX), *Y = drow(b, c, RY), *Z = drow(b, c, RZ),
                 *R = drow(b, c, RR);
    const bool px = !k.wall[0], py = !k.wall[1], pz = DIM == 3 && !k.wall[2];
    double tot = 0.0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
        const int i = PI[p], j = PJ[p];
        double dx = X[i] - X[j], dy = Y[i] - Y[j], dz = DIM == 3 ? Z[i] - Z[j] : 0.0;
        if (px) dx = min_image(dx, k.half_iv[0], k.iv[0]);
        if (py) dy = min_image(dy, k.half_iv[1], k.iv[1]);
        if (pz) dz = min_image(dz, k.half_iv[2], k.iv[2]);
        const double r1 = R[i], r2 = R[j];
        // pairs well apart (FP32, 1e-5) add nothing
        const float fx = ff_f32(dx), fy = ff_f32(dy), fz = DIM == 3 ? ff_f32(dz) : 0.f;
        const float fr = ff_f32(r1) + ff_f32(r2);
        if (fmaf(fz, fz, fmaf(fy, fy, fx * fx)) > fr * fr * (1.f + 1e-5f)) continue;
        double m = dx * dx + dy * dy;
        if (DIM == 3) m += dz * dz;
        double e = r1 + r2 - sqrt_d(m);
        if (e > 0) {
            e *= e;
            tot += 2.0 * e;
            if (per_bubble) {
                atomicAdd(b.energy + i, e);
                atomicAdd(b.energy + j, e);
            }
        }
    }
    const double t = block_reduce(tot, OpSum(), smem);
    if (threadIdx.x == 0) b.part[6 * gridDim.x + blockIdx.x] = t;
    if (last_block(&c->done[DC_MISC], gridDim.x)) {
        const double f = fold_partials(b.part + 6 * gridDim.x, gridDim.x, false, smem);
        if (threadIdx.x == 0) {
            c->misc_result = f;
            c->done[DC_MISC] = 0;
        }
    }
}

// calculateVolumes + sum, src/kernels.cu:1013-1024, src/simulator.cu:362-379
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_volume(Bufs b) {
    __shared__ double smem[32];
    Ctrl *c = b.ctrl;
    const int n = c->n;
    const double *R = drow(b, c, RR);
    double tot = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double radius = R[i];
        double volume = radius * radius * kPi;
        if (DIM == 3) volume *= radius * 1.33333333333333333333333333;
        tot += volume;
    }
    const double t = block_reduce(tot, OpSum(), smem);
    if (threadIdx.x == 0) b.part[6 * gridDim.x + blockIdx.x] = t;
    if (last_block(&c->done[DC_MISC], gridDim.x)) {
        const double f = fold_partials(b.part + 6 * gridDim.x, gridDim.x, false, smem);
        if (threadIdx.x == 0) {
            c->misc_result = f;
            c->done[DC_MISC] = 0;
        }
    }
}

}  // namespace

void launch_predict(const Launch &l, const Bufs &b, int dim) {
    if (dim == 3)
        CB_LAUNCH(l, k_predict, (<3>), wave_grid(k_predict<3>, l, l.step_bps), b);
    else
        CB_LAUNCH(l, k_predict, (<2>), wave_grid(k_predict<2>, l, l.step_bps), b);
}

// mode bits: 1 = gas exchange, 2 = flow. mode 0 is the bootstrap form.
void launch_pairs(const Launch &l, const Bufs &b, int dim, int mode) {
    const bool gas = mode & 1, flow = mode & 2;
#define CB_PAIRS(D, G, F) \
    CB_LAUNCH(l, k_pairs, (<D, G, F>), wave_grid(k_pairs<D, G, F>, l, l.pair_bps), b)
    if (dim == 3) {
        if (gas && flow) CB_PAIRS(3, true, true);
        else if (gas) CB_PAIRS(3, true, false);
        else if (flow) CB_PAIRS(3, false, true);
        else CB_PAIRS(3, false, false);
    } else {
        if (gas && flow) CB_PAIRS(2, true, true);
        else if (gas) CB_PAIRS(2, true, false);
        else if (flow) CB_PAIRS(2, false, true);
        else CB_PAIRS(2, false, false);
    }
#undef CB_PAIRS
}

void launch_correct(const Launch &l, const Bufs &b, int dim) {
    if (dim == 3)
        CB_LAUNCH(l, k_correct, (<3>), wave_grid(k_correct<3>, l, l.step_bps), b);
    else
        CB_LAUNCH(l, k_correct, (<2>), wave_grid(k_correct<2>, l, l.step_bps), b);
}

namespace {
template <int DIM, int BPS>
void launch_run_t(const RunLaunch &r, const Bufs &b, int mode) {
    const bool gas = mode & 1, flow = mode & 2;
    if (gas && flow) launch_coop(k_run<DIM, true, true, BPS>, r, b);
    else if (gas) launch_coop(k_run<DIM, true, false, BPS>, r, b);
    else if (flow) launch_coop(k_run<DIM, false, true, BPS>, r, b);
    else launch_coop(k_run<DIM, false, false, BPS>, r, b);
}
}  // namespace

void launch_run(const RunLaunch &r, const Bufs &b, int dim, int mode) {
    if (dim == 3)
        r.wide ? launch_run_t<3, kRunWide>(r, b, mode) : launch_run_t<3, kRunNarrow>(r, b, mode);
    else
        r.wide ? launch_run_t<2, kRunWide>(r, b, mode) : launch_run_t<2, kRunNarrow>(r, b, mode);
}

void launch_boot(const Launch &l, const Bufs &b, int dim, int phase) {
    if (dim == 3)
        k_boot<3><<<small_grid(l), kBlock, 0, l.stream>>>(b, phase);
    else
        k_boot<2><<<small_grid(l), kBlock, 0, l.stream>>>(b, phase);
    *l.launches += 1;
}

void launch_energy(const Launch &l, const Bufs &b, int dim, int per_bubble) {
    if (dim == 3)
        k_energy<3><<<small_grid(l, 4), kBlock, 0, l.stream>>>(b, per_bubble);
    else
        k_energy<2><<<small_grid(l, 4), kBlock, 0, l.stream>>>(b, per_bubble);
    *l.launches += 1;
}

void launch_volume(const Launch &l, const Bufs &b, int dim) {
    if (dim == 3)
        k_volume<3><<<small_grid(l), kBlock, 0, l.stream>>>(b);
    else
        k_volume<2><<<small_grid(l), kBlock, 0, l.stream>>>(b);
    *l.launches += 1;
}

}  // namespace cbg
