// FP64 DOP853 for one particle with a 2-D state.
//
// The method is the Dormand-Prince 8(5,3) pair with Hairer & Wanner's dop853
// step-size controller, which is what the reference's numbalsoda.dop853
// (called at integration.py:169-171) runs: HINIT initial step, error norm
// err5^2/(err5^2 + 0.01 err3^2) scaling, safe = 0.9, fac1 = 0.333, fac2 = 6,
// beta = 0, uround = 2.3e-16, no step-size increase right after a rejection.
//
// Arithmetic: every stage sum keeps the published operand order (ascending
// stage index, zero tableau entries skipped, stage 2 as (h*a21)*k1) and the
// file is compiled with -fmad=false, so results match the CPU oracle bit for
// bit apart from the library transcendentals of the analytic flows.
//
// Code shape: the twelve stages run as one rolled loop (the right-hand side is
// instantiated once per solver, not twelve times -- the unrolled form was
// instruction-fetch bound); stage derivatives live in this thread's column of
// shared memory and the tableau is a set of compile-time constants.  The
// derivative at the new point after an accepted step (FSAL) is the next step's
// stage 0.
//
// What bounds it: the FP64 pipe.  An FP64 add, multiply, FMA or compare of a
// warp takes 19 cycles of an SM (two lanes a cycle), as long as some 38
// integer instructions, so everything that is not the reference's own
// arithmetic -- zero tests, comparisons, sign handling -- stays off that pipe.
#pragma once

#include "detmath.h"
#include "dop853_tableau.h"
#include "nbcs_internal.cuh"

namespace nbcs {

constexpr int kThreads64 = 128;

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

// Comparison-based min/max (a NaN operand propagates the same way as in the
// CPU oracle; fmin/fmax would drop it).
__device__ __forceinline__ double dmin_(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ double dmax_(double a, double b) { return a > b ? a : b; }

// acc + c * k of a sum that starts at 0 (FIRST) or goes on: the product and
// the sum rounded separately.  The first term is one FMA with 0, whose single
// rounding is the product's.
template <bool FIRST>
__device__ __forceinline__ double dterm(double acc, double c, double k)
{
    return FIRST ? __fma_rn(c, k, 0.0) : acc + c * k;
}

// sum_{j < S} a_Sj k_j over the nonzero entries, in ascending j
template <int S, int KS, int J = 0, bool FIRST = true>
__device__ __forceinline__ void stage_terms64(const double2* kc, double& a0, double& a1)
{
    if constexpr (J < S) {
        constexpr double c = DP853D::a(S, J);
        if constexpr (c != 0.0) {
            const double2 kj = kc[J * KS];
            a0 = dterm<FIRST>(a0, c, kj.x);
            a1 = dterm<FIRST>(a1, c, kj.y);
            stage_terms64<S, KS, J + 1, false>(kc, a0, a1);
        } else {
            stage_terms64<S, KS, J + 1, FIRST>(kc, a0, a1);
        }
    }
}

// argument and time of stage S (a compile-time stage)
template <int S, int KS>
__device__ __forceinline__ void stage_arg64(const double2* kc, double h, const double* y,
                                            double* yy, double* c)
{
    if (S == 0) {
        yy[0] = y[0];
        yy[1] = y[1];
    } else if (S == 1) {
        const double2 k1 = kc[0];
        yy[0] = y[0] + h * DP853_A_2_1 * k1.x;
        yy[1] = y[1] + h * DP853_A_2_1 * k1.y;
    } else {
        double a0 = 0.0, a1 = 0.0;
        stage_terms64<S, KS>(kc, a0, a1);
        yy[0] = y[0] + h * a0;
        yy[1] = y[1] + h * a1;
    }
    *c = DP853D::c(S);
}

// the same for a runtime stage s that is uniform across the warp
template <int KS>
__device__ __forceinline__ void stage_arg64(int s, const double2* kc, double h, const double* y,
                                            double* yy, double* c)
{
    switch (s) {
    case 0: stage_arg64<0, KS>(kc, h, y, yy, c); break;
    case 1: stage_arg64<1, KS>(kc, h, y, yy, c); break;
    case 2: stage_arg64<2, KS>(kc, h, y, yy, c); break;
    case 3: stage_arg64<3, KS>(kc, h, y, yy, c); break;
    case 4: stage_arg64<4, KS>(kc, h, y, yy, c); break;
    case 5: stage_arg64<5, KS>(kc, h, y, yy, c); break;
    case 6: stage_arg64<6, KS>(kc, h, y, yy, c); break;
    case 7: stage_arg64<7, KS>(kc, h, y, yy, c); break;
    case 8: stage_arg64<8, KS>(kc, h, y, yy, c); break;
    case 9: stage_arg64<9, KS>(kc, h, y, yy, c); break;
    case 10: stage_arg64<10, KS>(kc, h, y, yy, c); break;
    default: stage_arg64<11, KS>(kc, h, y, yy, c); break;
    }
}

// sum b_j k_j and sum e5_j k_j over the stages with a nonzero weight (the
// first stage has both)
template <int KS, int J = 0>
__device__ __forceinline__ void step_sums64(const double2* kc, double* b, double* e5)
{
    if constexpr (J < 12) {
        constexpr double wb = DP853D::b(J), w5 = DP853D::e5(J);
        if constexpr (wb != 0.0 || w5 != 0.0) {
            const double2 kj = kc[J * KS];
            if constexpr (wb != 0.0) {
                b[0] = dterm<J == 0>(b[0], wb, kj.x);
                b[1] = dterm<J == 0>(b[1], wb, kj.y);
            }
            if constexpr (w5 != 0.0) {
                e5[0] = dterm<J == 0>(e5[0], w5, kj.x);
                e5[1] = dterm<J == 0>(e5[1], w5, kj.y);
            }
        }
        step_sums64<KS, J + 1>(kc, b, e5);
    }
}

// Order of nonnegative doubles (and +NaN above all) by their bit patterns: the
// comparisons of the step-size controller on the integer pipe, where an FP64
// compare takes 19 cycles of the FP64 pipe.
__device__ __forceinline__ unsigned long long dbits(double a)
{
    return (unsigned long long)__double_as_longlong(a);
}
__device__ __forceinline__ double min_nonneg(double a, double b) { return dbits(a) < dbits(b) ? a : b; }
__device__ __forceinline__ double max_nonneg(double a, double b) { return dbits(a) > dbits(b) ? a : b; }
// |a| with the sign of s
__device__ __forceinline__ double with_sign(double a, double s)
{
    return __longlong_as_double((long long)((dbits(a) & 0x7fffffffffffffffull) |
                                            (dbits(s) & 0x8000000000000000ull)));
}

struct Dop853Stats {
    int accepted, rejected, nfcn;
};

// Dense output (numbalsoda.dop853 with a t_eval grid: dop853's contd8 and its
// three extra stages) after the accepted step [xold, xold + h] from y0 to y1:
// stages k1, k6..k12 in slots 0, 5..11 of kc, the derivative at the end in
// slot 12; the extra stages go to slots 13..15.  Writes the interpolant at
// every due output time teval[*m] (up to the step's end) to dout[*m].
template <class Flow, int KS>
__device__ void dense_output64(const Flow& fl, const Params& P, double xold, double h,
                               const double* y0, const double* y1, double2* kc,
                               const double* __restrict__ teval, int n, int* m, double posneg,
                               double2* __restrict__ dout)
{
    double k[17][2];  // 1-based stages (only 1, 6..16 are used)
#pragma unroll
    for (int j = 6; j <= 13; ++j) {
        const double2 v = kc[(j - 1) * KS];
        k[j][0] = v.x;
        k[j][1] = v.y;
    }
    {
        const double2 v = kc[0];
        k[1][0] = v.x;
        k[1][1] = v.y;
    }
    double yy[2], kk[2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
        yy[i] = y0[i] + h * (DP853_A_14_1 * k[1][i] + DP853_A_14_7 * k[7][i]
                             + DP853_A_14_8 * k[8][i] + DP853_A_14_9 * k[9][i]
                             + DP853_A_14_10 * k[10][i] + DP853_A_14_11 * k[11][i]
                             + DP853_A_14_12 * k[12][i] + DP853_A_14_13 * k[13][i]);
    fl(xold + DP853_C_14 * h, yy, kk, P);
    k[14][0] = kk[0];
    k[14][1] = kk[1];
#pragma unroll
    for (int i = 0; i < 2; ++i)
        yy[i] = y0[i] + h * (DP853_A_15_1 * k[1][i] + DP853_A_15_6 * k[6][i]
                             + DP853_A_15_7 * k[7][i] + DP853_A_15_8 * k[8][i]
                             + DP853_A_15_11 * k[11][i] + DP853_A_15_12 * k[12][i]
                             + DP853_A_15_13 * k[13][i] + DP853_A_15_14 * k[14][i]);
    fl(xold + DP853_C_15 * h, yy, kk, P);
    k[15][0] = kk[0];
    k[15][1] = kk[1];
#pragma unroll
    for (int i = 0; i < 2; ++i)
        yy[i] = y0[i] + h * (DP853_A_16_1 * k[1][i] + DP853_A_16_6 * k[6][i]
                             + DP853_A_16_7 * k[7][i] + DP853_A_16_8 * k[8][i]
                             + DP853_A_16_9 * k[9][i] + DP853_A_16_13 * k[13][i]
                             + DP853_A_16_14 * k[14][i] + DP853_A_16_15 * k[15][i]);
    fl(xold + DP853_C_16 * h, yy, kk, P);
    k[16][0] = kk[0];
    k[16][1] = kk[1];
    double F[7][2];
#define NBCS_DENSE_ROW(r)                                                                      \
    (DP853_D_##r##_1 * k[1][i] + DP853_D_##r##_6 * k[6][i] + DP853_D_##r##_7 * k[7][i]       \
     + DP853_D_##r##_8 * k[8][i] + DP853_D_##r##_9 * k[9][i] + DP853_D_##r##_10 * k[10][i]   \
     + DP853_D_##r##_11 * k[11][i] + DP853_D_##r##_12 * k[12][i]                              \
     + DP853_D_##r##_13 * k[13][i] + DP853_D_##r##_14 * k[14][i]                              \
     + DP853_D_##r##_15 * k[15][i] + DP853_D_##r##_16 * k[16][i])
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double d = y1[i] - y0[i];
        F[0][i] = d;
        F[1][i] = h * k[1][i] - d;
        F[2][i] = 2.0 * d - h * (k[13][i] + k[1][i]);
        F[3][i] = h * NBCS_DENSE_ROW(4);
        F[4][i] = h * NBCS_DENSE_ROW(5);
        F[5][i] = h * NBCS_DENSE_ROW(6);
        F[6][i] = h * NBCS_DENSE_ROW(7);
    }
#undef NBCS_DENSE_ROW
    while (*m < n && (teval[*m] - (xold + h)) * posneg <= 0.0) {
        const double th = (teval[*m] - xold) / h, th1 = 1.0 - th;
        double o[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            double v = F[6][i] * th;
            v = (F[5][i] + v) * th1;
            v = (F[4][i] + v) * th;
            v = (F[3][i] + v) * th1;
            v = (F[2][i] + v) * th;
            v = (F[1][i] + v) * th1;
            v = (F[0][i] + v) * th;
            o[i] = v + y0[i];
        }
        dout[*m] = make_double2(o[0], o[1]);
        ++*m;
    }
}

// Integrate y over solver time [x, xend]; `kc` is this thread's shared-memory
// column of stage derivatives (stride KS, the block size).  Returns NBCS_PARTICLE_*.
// DENSE: also the positions at the n output times teval (teval[0] = x,
// teval[n-1] = xend) into dout[0 .. n), by dense output; kc needs 16 slots.
// When an output falls in an accepted step, the derivative at its end is
// evaluated there (for the interpolant) and handed to the next step as its
// first stage, with the same arguments as that stage would have had, so the
// step sequence is the one without outputs.
template <class Flow, int KS = kThreads64, bool DENSE = false>
__device__ int dop853_solve64(const Flow& fl, const Params& P, double x, double xend, double* y,
                              double rtol, double atol, int nmax, double2* kc, Dop853Stats* st,
                              const double* __restrict__ teval = nullptr, int n = 0,
                              double2* __restrict__ dout = nullptr)
{
    const double uround = 2.3e-16, safe = 0.9, facc1 = 1.0 / 0.333, facc2 = 1.0 / 6.0;
    const double posneg = (xend - x) >= 0.0 ? 1.0 : -1.0;
    const unsigned long long sgn = dbits(posneg) & 0x8000000000000000ull;
    double yy[2], kk[2], h = 0.0, hnew, hmax, err, err2, deno, fac, sk, erri, sqr;
    bool last = false, reject = false;
    int nstep = 0, status = NBCS_PARTICLE_OK;
    int m = 1;  // next dense output
    st->accepted = st->rejected = st->nfcn = 0;
    if (DENSE) dout[0] = make_double2(y[0], y[1]);
    if (xend == x) {
        if (DENSE)
            for (; m < n; ++m) dout[m] = make_double2(y[0], y[1]);
        return NBCS_PARTICLE_OK;
    }
    hmax = fabs(xend - x);

    // HINIT (f0 = f(x, y) is also stage 0 of the first step); one RHS site
    double f0[2] = {0.0, 0.0}, dnf = 0.0, dny = 0.0;
#pragma unroll 1
    for (int e = 0; e < 2; ++e) {
#pragma unroll
        for (int i = 0; i < 2; ++i) yy[i] = e ? y[i] + h * f0[i] : y[i];
        fl(e ? x + h : x, yy, kk, P);
        if (e == 0) {
            f0[0] = kk[0];
            f0[1] = kk[1];
            kc[0] = make_double2(kk[0], kk[1]);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                sk = atol + rtol * fabs(y[i]);
                sqr = f0[i] / sk;
                dnf += sqr * sqr;
                sqr = y[i] / sk;
                dny += sqr * sqr;
            }
            if (dnf <= 1.0e-10 || dny <= 1.0e-10) h = 1.0e-6;
            else h = sqrt(dny / dnf) * 0.01;
            h = dmin_(h, hmax);
            h = posneg >= 0.0 ? fabs(h) : -fabs(h);
        } else {
            double der2 = 0.0, der12, h1;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                sk = atol + rtol * fabs(y[i]);
                sqr = (kk[i] - f0[i]) / sk;
                der2 += sqr * sqr;
            }
            der2 = sqrt(der2) / h;
            der12 = dmax_(fabs(der2), sqrt(dnf));
            if (der12 <= 1.0e-15) h1 = dmax_(1.0e-6, fabs(h) * 1.0e-3);
            else h1 = nbcs_root8(0.01 / der12);  // (0.01/der12)^(1/8)
            h = dmin_(100.0 * fabs(h), dmin_(h1, hmax));
            h = posneg >= 0.0 ? fabs(h) : -fabs(h);
        }
    }
    st->nfcn += 2;

    bool fsal = false;  // stage 0 (the derivative at the new point) still to evaluate
    for (;;) {
        if (nstep > nmax) { status = NBCS_PARTICLE_MAX_STEPS; break; }
        if (dbits(0.1 * fabs(h)) <= dbits(fabs(x) * uround)) {
            status = NBCS_PARTICLE_STEP_UNDERFLOW;
            break;
        }
        // beyond xend in the direction of the integration
        if ((long long)(dbits(x + 1.01 * h - xend) ^ sgn) > 0) {
            h = xend - x;
            last = true;
        }
        nstep++;
        // every lane counts the stages from 0 (a rejected step skips stage 0,
        // whose derivative is still valid): the stage index is warp-uniform
#pragma unroll 1
        for (int s = 0; s < 12; ++s) {
            if (s == 0 && !fsal) continue;
            double cs;
            stage_arg64<KS>(s, kc, h, y, yy, &cs);
            fl(x + cs * h, yy, kk, P);
            kc[s * KS] = make_double2(kk[0], kk[1]);
        }
        fsal = false;
        st->nfcn += 11;
        double b[2] = {0.0, 0.0}, e5[2] = {0.0, 0.0}, ynew[2];
        step_sums64<KS>(kc, b, e5);
        const double2 k1 = kc[0], k9 = kc[8 * KS], k12 = kc[11 * KS];
        const double k1v[2] = {k1.x, k1.y}, k9v[2] = {k9.x, k9.y}, k12v[2] = {k12.x, k12.y};
        err = 0.0;
        err2 = 0.0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            ynew[i] = y[i] + h * b[i];
            sk = atol + rtol * max_nonneg(fabs(y[i]), fabs(ynew[i]));
            erri = b[i] - DP853_BHH1 * k1v[i] - DP853_BHH2 * k9v[i] - DP853_BHH3 * k12v[i];
            sqr = erri / sk;
            err2 += sqr * sqr;
            sqr = e5[i] / sk;
            err += sqr * sqr;
        }
        deno = err + 0.01 * err2;
        if (dbits(deno) == 0ull) deno = 1.0;
        err = fabs(h) * err * sqrt(1.0 / (deno * 2.0));
        if (dbits(fabs(err)) > 0x7ff0000000000000ull) {  // NaN
            status = NBCS_PARTICLE_NONFINITE;
            break;
        }
        // err^(1/8); beta = 0: the Lund factor facold^beta is 1.  A rejected
        // step's h / min(facc1, fac11 / safe) is the same quotient: there
        // fac11 / safe is above facc2.
        fac = max_nonneg(facc2, min_nonneg(facc1, nbcs_root8(err) / safe));
        hnew = h / fac;
        if (dbits(err) <= 0x3ff0000000000000ull) {  // err <= 1
            st->accepted++;
            st->nfcn++;  // the derivative at the new point (next step's stage 0)
            bool have_end_derivative = false;
            if (DENSE && m < n && (teval[m] - (x + h)) * posneg <= 0.0) {
                fl(x + h, ynew, kk, P);
                kc[12 * KS] = make_double2(kk[0], kk[1]);
                dense_output64<Flow, KS>(fl, P, x, h, y, ynew, kc, teval, n, &m, posneg, dout);
                kc[0] = make_double2(kk[0], kk[1]);
                st->nfcn += 3;
                have_end_derivative = true;
            }
            y[0] = ynew[0];
            y[1] = ynew[1];
            x = x + h;
            fsal = !have_end_derivative;
            if (last) break;
            hnew = with_sign(min_nonneg(fabs(hnew), reject ? min_nonneg(hmax, fabs(h)) : hmax), posneg);
            reject = false;
        } else {
            reject = true;
            if (st->accepted >= 1) st->rejected++;
            last = false;
        }
        h = hnew;
    }
    return status;
}

}  // namespace nbcs
