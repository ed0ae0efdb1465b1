// FP64 DOP853 for one particle with a 2-D state.
//
// The method is the Dormand-Prince 8(5,3) pair with Hairer & Wanner's dop853
// step-size controller, which is what the reference's numbalsoda.dop853
// (called at integration.py:169-171) runs: HINIT initial step, error norm
// err5^2/(err5^2 + 0.01 err3^2) scaling, safe = 0.9, fac1 = 0.333, fac2 = 6,
// beta = 0, uround = 2.3e-16, no step-size increase right after a rejection.
//
// Arithmetic: every stage sum keeps the published operand order (ascending
// stage index, zero tableau entries skipped, stage 2 as (h*a21)*k1), every
// product and sum rounded separately (the file is compiled with -fmad=false),
// so results match the CPU oracle bit for bit apart from the transcendentals of
// the analytic flows.
//
// Work split: two adjacent lanes integrate one particle, lane q its component
// q.  Everything that is per component -- stage sums, the step, its error, the
// dense output, half of the right-hand side -- is one instruction for both; the
// step-size control works on values that both lanes hold.  Against one thread a
// particle this halves what a warp has to do before it is done, which is what
// small and middling grids wait for: 42,588 particles are 9 warps an SM of one
// thread a particle -- 3, 2, 2, 2 on its four partitions, whose FP64 units do
// not help one another out.
//
// What bounds it: the FP64 pipe.  An FP64 add, multiply, FMA or compare of a
// warp takes 19 cycles of an SM (two lanes a cycle), as long as some 38
// integer instructions.  So products, quotients and roots run on the integer
// pipe (intfp64.h: correctly rounded, the same bits), and the FP64 pipe has the
// sums.  Sums of products test once, at their end, whether every operand was in
// the integer arithmetic's range, and are redone on the FP64 pipe if not (a
// derivative of exactly zero, on a wall say): a test per product costs half as
// much again and keeps the products from overlapping.
// Flow maps with one lane a particle and all arithmetic on the FP64 pipe, and
// as it is: double gyre 401 x 201 5.45 -> 2.75 ms, 21 x 11 1.02 -> 0.64 ms;
// geophysical flow 338 x 126 at rtol 1e-6 31.3 -> 22.1 ms, where the FP64 pipe
// is busy 79 % of the time (143 operations an evaluation and lane pair).
//
// Code shape: integer arithmetic is many instructions, and what a step runs
// through has to stay in the instruction caches (with the stage sums unrolled
// and two copies of the right-hand side, waiting for instructions was the
// largest stall).  So the stages are one rolled loop, HINIT's evaluations are
// two more of its stages, the sums run over tables in constant memory, and the
// step-size control calls its roots and quotients.  Stage derivatives live in
// this thread's column of shared memory.  The derivative at the new point after
// an accepted step (FSAL) is the next step's stage 0.
#pragma once

#include "detmath.h"
#include "dop853_tableau.h"
#include "intfp64.h"
#include "nbcs_internal.cuh"

namespace nbcs {

constexpr int kThreads64 = 128;

// the other component's value of the same particle
__device__ __forceinline__ unsigned pair_mask64() { return 3u << (threadIdx.x & 30u); }
__device__ __forceinline__ double other64(double v)
{
    return __shfl_xor_sync(pair_mask64(), v, 1);
}

// DP853 tableau as compile-time values, 0-based stage index: stage s uses a(s, j)
// for j < s.  As constants of the compiler (not of a memory bank) the zero
// entries cost nothing; tested at run time each of them cost an FP64 compare,
// 19 cycles of the SM's FP64 pipe (90 a step).
struct DP853D {
    __host__ __device__ static constexpr double a(int s, int j)
    {
        constexpr double t[12][12] = {
            {0.0},
            {DP853_A_2_1},
            {DP853_A_3_1, DP853_A_3_2},
            {DP853_A_4_1, DP853_A_4_2, DP853_A_4_3},
            {DP853_A_5_1, DP853_A_5_2, DP853_A_5_3, DP853_A_5_4},
            {DP853_A_6_1, DP853_A_6_2, DP853_A_6_3, DP853_A_6_4, DP853_A_6_5},
            {DP853_A_7_1, DP853_A_7_2, DP853_A_7_3, DP853_A_7_4, DP853_A_7_5, DP853_A_7_6},
            {DP853_A_8_1, DP853_A_8_2, DP853_A_8_3, DP853_A_8_4, DP853_A_8_5, DP853_A_8_6,
             DP853_A_8_7},
            {DP853_A_9_1, DP853_A_9_2, DP853_A_9_3, DP853_A_9_4, DP853_A_9_5, DP853_A_9_6,
             DP853_A_9_7, DP853_A_9_8},
            {DP853_A_10_1, DP853_A_10_2, DP853_A_10_3, DP853_A_10_4, DP853_A_10_5, DP853_A_10_6,
             DP853_A_10_7, DP853_A_10_8, DP853_A_10_9},
            {DP853_A_11_1, DP853_A_11_2, DP853_A_11_3, DP853_A_11_4, DP853_A_11_5, DP853_A_11_6,
             DP853_A_11_7, DP853_A_11_8, DP853_A_11_9, DP853_A_11_10},
            {DP853_A_12_1, DP853_A_12_2, DP853_A_12_3, DP853_A_12_4, DP853_A_12_5, DP853_A_12_6,
             DP853_A_12_7, DP853_A_12_8, DP853_A_12_9, DP853_A_12_10, DP853_A_12_11},
        };
        return t[s][j];
    }
    __host__ __device__ static constexpr double c(int s)
    {
        constexpr double t[12] = {0.0, DP853_C_2, DP853_C_3, DP853_C_4, DP853_C_5, DP853_C_6,
                                  DP853_C_7, DP853_C_8, DP853_C_9, DP853_C_10, DP853_C_11, 1.0};
        return t[s];
    }
    __host__ __device__ static constexpr double b(int j)
    {
        constexpr double t[12] = {DP853_B_1, DP853_B_2, DP853_B_3, DP853_B_4, DP853_B_5,
                                  DP853_B_6, DP853_B_7, DP853_B_8, DP853_B_9, DP853_B_10,
                                  DP853_B_11, DP853_B_12};
        return t[j];
    }
    __host__ __device__ static constexpr double e5(int j)
    {
        constexpr double t[12] = {DP853_E5_1, DP853_E5_2, DP853_E5_3, DP853_E5_4, DP853_E5_5,
                                  DP853_E5_6, DP853_E5_7, DP853_E5_8, DP853_E5_9, DP853_E5_10,
                                  DP853_E5_11, DP853_E5_12};
        return t[j];
    }
};

// Operand ranges of a group of integer products: note64 gathers them, fits64
// tells whether all were in range.
__device__ __forceinline__ unsigned note64(double a)
{
    return (unsigned)__double2hiint(a) - 0x30000000u;
}
__device__ __forceinline__ bool fits64(unsigned notes) { return (notes & 0x60000000u) == 0; }

template <bool FIT>
__device__ __forceinline__ double mul64(double a, double b)
{
    return FIT ? ip_mul_fit(a, b) : a * b;
}

// Stage coefficients in the order of their use -- entry o of stage s is its o-th
// nonzero a_sj, with j -- and the stages with a weight in the step's sums (all
// of them have e5_j, some no b_j).  A zero ends a list.
struct Term64 {
    double c;
    int j, pad;
};
struct Tables64 {
    Term64 a[12][12];
    double c[12];
    double b[9], e5[9];
    int j[9];
};

constexpr Tables64 tables64()
{
    Tables64 t = {};
    int n = 0;
    for (int s = 0; s < 12; ++s) {
        int o = 0;
        for (int j = 0; j < s; ++j)
            if (DP853D::a(s, j) != 0.0) t.a[s][o++] = {DP853D::a(s, j), j, 0};
        t.c[s] = DP853D::c(s);
        if (DP853D::e5(s) != 0.0) {
            t.j[n] = s;
            t.b[n] = DP853D::b(s);
            t.e5[n++] = DP853D::e5(s);
        }
    }
    return t;
}

static __constant__ Tables64 kT64 = tables64();
// whether a double is zero, from its high half (the constants here are normal)
__device__ __forceinline__ bool none64(double c) { return __double2hiint(c) == 0; }

// acc + c k of a sum that starts at 0 (first) or goes on; on the FP64 pipe the
// first product is rounded in an FMA with the 0
template <bool FIT>
__device__ __forceinline__ double sum64(double acc, double c, double k, bool first)
{
    if (!FIT) return first ? __fma_rn(c, k, 0.0) : acc + c * k;
    const double p = ip_mul_fit(c, k);
    return first ? p : acc + p;
}

// Argument and time of stage s (uniform across the warp).  False when an
// operand did not fit the integer arithmetic.  The sum is a rolled loop:
// unrolled, the fifty products of a step are 20 KB of code.
template <bool FIT, int KS>
__device__ __forceinline__ bool stage_arg64(int s, const double* kc, double x, double h, double y,
                                            double* yy, double* t)
{
    unsigned notes = note64(h);
    *t = x + (s == 11 ? h : mul64<FIT>(kT64.c[s], h));
    if (s == 1) {
        const double k1 = kc[0], ha = mul64<FIT>(h, DP853_A_2_1);
        notes |= note64(k1);
        *yy = y + mul64<FIT>(ha, k1);
    } else {
        double a = 0.0;
#pragma unroll 1
        for (int o = 0; !none64(kT64.a[s][o].c); ++o) {
            const double c = kT64.a[s][o].c, k = kc[kT64.a[s][o].j * KS];
            notes |= note64(k);
            a = sum64<FIT>(a, c, k, o == 0);
        }
        notes |= note64(a);
        *yy = y + mul64<FIT>(h, a);
    }
    return fits64(notes);
}

// The step's increment b, the two error sums e3 and e5 and the new position;
// false when an operand did not fit.
template <bool FIT, int KS>
__device__ __forceinline__ bool step_sums64(const double* kc, double h, double y, double* ynew,
                                            double* e3, double* e5)
{
    unsigned notes = note64(h);
    double b = 0.0, e = 0.0;
#pragma unroll 1
    for (int o = 0; !none64(kT64.e5[o]); ++o) {
        const double k = kc[kT64.j[o] * KS];
        notes |= note64(k);
        if (!none64(kT64.b[o])) b = sum64<FIT>(b, kT64.b[o], k, o == 0);
        e = sum64<FIT>(e, kT64.e5[o], k, o == 0);
    }
    notes |= note64(b);
    *ynew = y + mul64<FIT>(h, b);
    *e3 = b - mul64<FIT>(DP853_BHH1, kc[0]) - mul64<FIT>(DP853_BHH2, kc[8 * KS]) -
          mul64<FIT>(DP853_BHH3, kc[11 * KS]);
    *e5 = e;
    return fits64(notes);
}

static_assert(DP853D::b(0) != 0.0 && DP853D::e5(0) != 0.0, "the first stage has both weights");

// Order of nonnegative doubles (and +NaN above all) by their bit patterns: the
// comparisons of the step-size controller on the integer pipe.
__device__ __forceinline__ unsigned long long dbits(double a)
{
    return (unsigned long long)__double_as_longlong(a);
}
__device__ __forceinline__ double min_nonneg(double a, double b) { return dbits(a) < dbits(b) ? a : b; }
__device__ __forceinline__ double max_nonneg(double a, double b) { return dbits(a) > dbits(b) ? a : b; }
// |a| with the sign of s
__device__ __forceinline__ double with_sign(double a, double s)
{
    return __hiloint2double((__double2hiint(a) & 0x7fffffff) | (__double2hiint(s) & (int)0x80000000u),
                            __double2loint(a));
}
__device__ __forceinline__ double abs64(double a)
{
    return __hiloint2double(__double2hiint(a) & 0x7fffffff, __double2loint(a));
}

// a / b, sqrt and a / 0.9 of the step-size control: once or a few times a step,
// so one copy of each (the loop's code has to stay in the instruction caches)
static __device__ __noinline__ double quot64(double a, double b) { return ip_div(a, ip_reciprocal(b)); }
static __device__ __noinline__ double root64(double x) { return ip_sqrt(x); }
static __device__ __noinline__ double prod64(double a, double b) { return ip_mul(a, b); }
// sum of the two components' squares of v / s (the order does not matter)
__device__ __forceinline__ double norm2_64(double v, double s)
{
    const double q = quot64(v, s), q2 = prod64(q, q);
    return q2 + other64(q2);
}

struct Dop853Stats {
    int accepted, rejected, nfcn;
};

// Dense output (numbalsoda.dop853 with a t_eval grid: dop853's contd8 and its
// three extra stages) after the accepted step [xold, xold + h] from y0 to y1:
// stages k1, k6..k12 in slots 0, 5..11 of kc; the derivative at the end goes to
// slot 12, the extra stages to slots 13..15.  Writes the interpolant at every
// due output time teval[*m] (up to the step's end) to dout[2 * *m] (this lane's
// component).
template <class Flow, int KS>
__device__ void dense_output64(const Flow& fl, const Params& P, double xold, double h, double y0,
                               double y1, double* kc, int q, const double* __restrict__ teval,
                               int n, int* m, double posneg, double* __restrict__ dout)
{
#define K_(j) kc[(j - 1) * KS]
#pragma unroll 1
    for (int s = 13; s <= 16; ++s) {
        double yy, t;
        if (s == 13) {
            yy = y1;
            t = xold + h;
        } else if (s == 14) {
            yy = y0 + h * (DP853_A_14_1 * K_(1) + DP853_A_14_7 * K_(7) + DP853_A_14_8 * K_(8)
                           + DP853_A_14_9 * K_(9) + DP853_A_14_10 * K_(10)
                           + DP853_A_14_11 * K_(11) + DP853_A_14_12 * K_(12)
                           + DP853_A_14_13 * K_(13));
            t = xold + DP853_C_14 * h;
        } else if (s == 15) {
            yy = y0 + h * (DP853_A_15_1 * K_(1) + DP853_A_15_6 * K_(6) + DP853_A_15_7 * K_(7)
                           + DP853_A_15_8 * K_(8) + DP853_A_15_11 * K_(11)
                           + DP853_A_15_12 * K_(12) + DP853_A_15_13 * K_(13)
                           + DP853_A_15_14 * K_(14));
            t = xold + DP853_C_15 * h;
        } else {
            yy = y0 + h * (DP853_A_16_1 * K_(1) + DP853_A_16_6 * K_(6) + DP853_A_16_7 * K_(7)
                           + DP853_A_16_8 * K_(8) + DP853_A_16_9 * K_(9)
                           + DP853_A_16_13 * K_(13) + DP853_A_16_14 * K_(14)
                           + DP853_A_16_15 * K_(15));
            t = xold + DP853_C_16 * h;
        }
        K_(s) = fl(t, yy, q, P);
    }
    double F[7];
#define NBCS_DENSE_ROW(r)                                                                      \
    (DP853_D_##r##_1 * K_(1) + DP853_D_##r##_6 * K_(6) + DP853_D_##r##_7 * K_(7)              \
     + DP853_D_##r##_8 * K_(8) + DP853_D_##r##_9 * K_(9) + DP853_D_##r##_10 * K_(10)          \
     + DP853_D_##r##_11 * K_(11) + DP853_D_##r##_12 * K_(12) + DP853_D_##r##_13 * K_(13)      \
     + DP853_D_##r##_14 * K_(14) + DP853_D_##r##_15 * K_(15) + DP853_D_##r##_16 * K_(16))
    const double d = y1 - y0;
    F[0] = d;
    F[1] = h * K_(1) - d;
    F[2] = 2.0 * d - h * (K_(13) + K_(1));
    F[3] = h * NBCS_DENSE_ROW(4);
    F[4] = h * NBCS_DENSE_ROW(5);
    F[5] = h * NBCS_DENSE_ROW(6);
    F[6] = h * NBCS_DENSE_ROW(7);
#undef NBCS_DENSE_ROW
#undef K_
    while (*m < n && (teval[*m] - (xold + h)) * posneg <= 0.0) {
        const double th = (teval[*m] - xold) / h, th1 = 1.0 - th;
        double v = F[6] * th;
        v = (F[5] + v) * th1;
        v = (F[4] + v) * th;
        v = (F[3] + v) * th1;
        v = (F[2] + v) * th;
        v = (F[1] + v) * th1;
        v = (F[0] + v) * th;
        dout[2 * *m] = v + y0;
        ++*m;
    }
}

// Integrate component q of a particle (the pair's other lane has the other one;
// the two call together) from *yp over solver time [x, xend]; `kc` is this
// thread's shared-memory column of stage derivatives (stride KS, the block
// size).  Returns NBCS_PARTICLE_*, the same on both lanes.
// DENSE: also the positions at the n output times teval (teval[0] = x,
// teval[n-1] = xend) into dout[0], dout[2] .. dout[2 (n-1)], by dense output;
// kc needs 16 slots.  When an output falls in an accepted step, the derivative
// at its end is evaluated there (for the interpolant) and handed to the next
// step as its first stage, with the same arguments as that stage would have
// had, so the step sequence is the one without outputs.
// FEW: the launch has too few warps for the pipes to fill; then what counts is
// a warp's own latency, and a product on the FP64 pipe has half the integer
// one's.
template <class Flow, int KS = kThreads64, bool DENSE = false, bool FEW = false>
__device__ int dop853_solve64(const Flow& fl, const Params& P, double x, double xend, double* yp,
                              int q, double rtol, double atol, int nmax, double* kc,
                              Dop853Stats* st, const double* __restrict__ teval = nullptr,
                              int n = 0, double* __restrict__ dout = nullptr)
{
    const double uround = 2.3e-16, facc1 = 1.0 / 0.333, facc2 = 1.0 / 6.0;
    const double posneg = (xend - x) >= 0.0 ? 1.0 : -1.0;
    const unsigned long long sgn = dbits(posneg) & 0x8000000000000000ull;
    double y = *yp, h = 0.0, hnew, err, err2, deno;
    bool last = false, reject = false;
    int nstep = 0, status = NBCS_PARTICLE_OK;
    int m = 1;  // next dense output
    st->accepted = st->rejected = st->nfcn = 0;
    if (DENSE) dout[0] = y;
    if (xend == x) {
        if (DENSE)
            for (; m < n; ++m) dout[2 * m] = y;
        return NBCS_PARTICLE_OK;
    }
    const double hmax = fabs(xend - x);

    // The right-hand side is called at one site (its code has to stay in the
    // instruction caches): stages 12 and 13 are HINIT's two evaluations, f0 =
    // f(x, y), which is also stage 0 of the first step, and the Euler probe.
    int s0 = 12, s1 = 14;
    double dnf = 0.0;
    const double sk0 = atol + rtol * abs64(y);
    bool fsal = false;  // stage 0 (the derivative at the new point) still to evaluate
    for (;;) {
        if (s0 == 0) {
            if (nstep > nmax) { status = NBCS_PARTICLE_MAX_STEPS; break; }
            const unsigned long long least = dbits(abs64(x) * uround);
            // (a NaN on either side, of a NaN start time say, is no underflow)
            if (dbits(0.1 * abs64(h)) <= least && least <= 0x7ff0000000000000ull) {
                status = NBCS_PARTICLE_STEP_UNDERFLOW;
                break;
            }
            // beyond xend in the direction of the integration: above zero, not NaN
            if ((dbits(x + 1.01 * h - xend) ^ sgn) - 1ull < 0x7ff0000000000000ull) {
                h = xend - x;
                last = true;
            }
            nstep++;
        }
        // every lane counts the stages from 0 (a rejected step skips stage 0,
        // whose derivative is still valid): the stage index is warp-uniform
#pragma unroll 1
        for (int s = s0; s < s1; ++s) {
            if (s == 0 && !fsal) continue;
            double yy = y, t = x;
            if (s == 13) {
                yy = y + h * kc[0];
                t = x + h;
            } else if (s > 0 && s < 12) {
                if (FEW || !stage_arg64<true, KS>(s, kc, x, h, y, &yy, &t))
                    stage_arg64<false, KS>(s, kc, x, h, y, &yy, &t);
            }
            const double kk = fl(t, yy, q, P);
            if (s < 12) {
                kc[s * KS] = kk;
            } else if (s == 12) {
                kc[0] = kk;
                dnf = norm2_64(kk, sk0);
                const double dny = norm2_64(y, sk0);
                if (dnf <= 1.0e-10 || dny <= 1.0e-10) h = 1.0e-6;
                else h = root64(quot64(dny, dnf)) * 0.01;
                h = h < hmax ? h : hmax;  // a NaN hmax stays
                h = with_sign(h, posneg);
            } else {
                const double der2 = root64(norm2_64(kk - kc[0], sk0)) / h;
                const double f = root64(dnf), der12 = fabs(der2) > f ? fabs(der2) : f;
                double h1;
                if (der12 <= 1.0e-15) h1 = 1.0e-6 > fabs(h) * 1.0e-3 ? 1.0e-6 : fabs(h) * 1.0e-3;
                else h1 = root64(root64(root64(0.01 / der12)));  // (0.01/der12)^(1/8)
                h1 = h1 < hmax ? h1 : hmax;
                h = 100.0 * fabs(h) < h1 ? 100.0 * fabs(h) : h1;
                h = with_sign(h, posneg);
            }
        }
        if (s0) {
            st->nfcn += 2;
            s0 = 0;
            s1 = 12;
            continue;
        }
        fsal = false;
        st->nfcn += 11;
        double ynew, e3, e5;
        if (FEW || !step_sums64<true, KS>(kc, h, y, &ynew, &e3, &e5))
            step_sums64<false, KS>(kc, h, y, &ynew, &e3, &e5);
        const double sk = atol + prod64(rtol, max_nonneg(abs64(y), abs64(ynew)));
        err2 = norm2_64(e3, sk);
        err = norm2_64(e5, sk);
        deno = err + 0.01 * err2;
        if (ip_zero(deno)) deno = 1.0;
        err = prod64(prod64(abs64(h), err), root64(quot64(1.0, 2.0 * deno)));
        if (dbits(abs64(err)) > 0x7ff0000000000000ull) {  // NaN
            status = NBCS_PARTICLE_NONFINITE;
            break;
        }
        // err^(1/8); beta = 0: the Lund factor facold^beta is 1.  A rejected
        // step's h / min(facc1, fac11 / safe) is the same quotient: there
        // fac11 / safe is above facc2.
        const double fac11 = root64(root64(root64(err)));
        hnew = quot64(h, max_nonneg(facc2, min_nonneg(facc1, quot64(fac11, 0.9))));
        if (dbits(err) <= 0x3ff0000000000000ull) {  // err <= 1
            st->accepted++;
            st->nfcn++;  // the derivative at the new point (next step's stage 0)
            bool have_end_derivative = false;
            if (DENSE && m < n && (teval[m] - (x + h)) * posneg <= 0.0) {
                dense_output64<Flow, KS>(fl, P, x, h, y, ynew, kc, q, teval, n, &m, posneg, dout);
                kc[0] = kc[12 * KS];
                st->nfcn += 3;
                have_end_derivative = true;
            }
            y = ynew;
            x = x + h;
            fsal = !have_end_derivative;
            if (last) break;
            hnew = with_sign(min_nonneg(abs64(hnew), reject ? min_nonneg(hmax, abs64(h)) : hmax),
                             posneg);
            reject = false;
        } else {
            reject = true;
            if (st->accepted >= 1) st->rejected++;
            last = false;
        }
        h = hnew;
    }
    *yp = y;
    return status;
}

}  // namespace nbcs
