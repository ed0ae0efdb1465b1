// FP64 device right-hand sides.
//
// These restate the reference's numba @cfunc bodies operation for operation
// (same operand order, every + - * / separately rounded: this file is only
// compiled with -fmad=false), so that with the same inputs they produce the
// same doubles as the CPU oracle apart from the last-bit differences of the
// transcendental functions.
//
//   double gyre   flows.py:1146-1158
//   Bickley jet   flows.py:1182-1213
//   spline RHS    flows.py:154-254 (interpolation.eval_spline, k=3)
#pragma once

#include "detmath.h"
#include "intfp64.h"
#include "nbcs_internal.cuh"

namespace nbcs {

#define NBCS_PI 3.141592653589793

struct FlowDG64 {
    __device__ __forceinline__ void operator()(double t, const double* y, double* dy,
                                               const Params& P) const
    {
        const double* p = P.v;
        double tt = p[0] * t;
        double a = p[2] * sin(p[4] * tt + p[5]);
        double b = 1.0 - 2.0 * a;
        double f = a * (y[0] * y[0]) + b * y[0];
        double df = 2.0 * a * y[0] + b;
        double sf, cf, sy, cy;
        sincos(NBCS_PI * f, &sf, &cf);
        sincos(NBCS_PI * y[1], &sy, &cy);
        dy[0] = p[0] * (-NBCS_PI * p[1] * sf * cy - p[3] * y[0]);
        dy[1] = p[0] * (NBCS_PI * p[1] * cf * sy * df - p[3] * y[1]);
    }
};

struct FlowBickley64 {
    __device__ __forceinline__ void operator()(double t, const double* y, double* dy,
                                               const Params& P) const
    {
        const double* p = P.v;
        double tt = p[0] * t;
        double Y = y[1] / p[2];
        double ch = cosh(Y);
        double sech2 = 1.0 / (ch * ch);
        double s1 = y[0] - p[9] * tt, s2 = y[0] - p[10] * tt, s3 = y[0] - p[11] * tt;
        double sn1, cs1, sn2, cs2, sn3, cs3;
        sincos(p[6] * s1, &sn1, &cs1);
        sincos(p[7] * s2, &sn2, &cs2);
        sincos(p[8] * s3, &sn3, &cs3);
        dy[0] = p[0] * (p[1] * sech2 + 2.0 * p[1] * tanh(Y) * sech2
                                           * (p[3] * cs1 + p[4] * cs2 + p[5] * cs3));
        dy[1] = -p[0] * (p[1] * p[2] * sech2
                         * (p[3] * p[6] * sn1 + p[4] * p[7] * sn2 + p[5] * p[8] * sn3));
    }
};

// Python's float modulo a % 360 (sign of the divisor), as numba evaluates it.
// For |a| < 360 -- every longitude that does not lap the globe within a stage
// -- fmod returns its argument; the range test is on the bit pattern.
__device__ __forceinline__ double py_mod360(double a)
{
    const unsigned hi = (unsigned)(__double_as_longlong(a) >> 32);
    double m = a;
    if ((hi & 0x7fffffffu) >= 0x40768000u) m = fmod(a, 360.0);  // |a| >= 360, inf, NaN
    const long long mb = __double_as_longlong(m);
    if (ip_zero(m)) return 0.0;
    return mb < 0 ? m + 360.0 : m;  // NaN stays NaN
}

// Weights of the four cubic B-spline pieces at offset t:
//   w0 = (-1/6) t^3 + (3/6) t^2 + (-3/6) t + (1/6)
//   w1 =  (3/6) t^3 + (-6/6) t^2 + (0/6) t + (4/6)
//   w2 = (-3/6) t^3 + (3/6) t^2 + (3/6) t + (1/6)
//   w3 =  (1/6) t^3 + 0 + 0 + 0
// in the reference's operation order.  Products with 1/2 and 1 are exact, so
// they ride in the FMA of the sum that follows (one rounding, the sum's), the
// zero terms fall away (t is finite or NaN), and w2's two halvings become one
// of the sum: 11 FP64 operations for 27, the same bits.
__device__ __forceinline__ void bspline_w64(double t, double* w)
{
    const double t2 = t * t, t3 = t2 * t, s3 = (1.0 / 6.0) * t3;
    w[0] = __fma_rn(-0.5, t, __fma_rn(0.5, t2, -s3)) + 1.0 / 6.0;
    w[1] = __fma_rn(0.5, t3, -t2) + 4.0 / 6.0;
    w[2] = __fma_rn(0.5, (t2 - t3) + t, 1.0 / 6.0);
    w[3] = s3;
}

// derivative of the basis with respect to the offset t
__device__ __forceinline__ void bspline_dw64(double t, double* w)
{
    double t2 = t * t;
    w[0] = (-3.0 / 6.0) * t2 + (6.0 / 6.0) * t + (-3.0 / 6.0);
    w[1] = (9.0 / 6.0) * t2 + (-12.0 / 6.0) * t + (0.0 / 6.0);
    w[2] = (-9.0 / 6.0) * t2 + (6.0 / 6.0) * t + (3.0 / 6.0);
    w[3] = (3.0 / 6.0) * t2 + (0.0 / 6.0) * t + (0.0 / 6.0);
}

// Cell index and fractional offset along axis d of a coordinate x; dx = x - a.
// A coordinate beyond the far end b sets *outside (it can only lie in the last
// cell, so the other cells skip the compare); a NaN coordinate takes any cell
// (and a NaN offset).  floor() runs beside the FP64 pipe; the cell index comes
// from the bits of its result, where the conversions to int and back and the
// two range compares took four FP64-pipe slots an axis.
__device__ __forceinline__ int spline_locate64(const SplineGrid& g, int d, double x, double dx,
                                               double* t, bool* outside)
{
    const double u = dx * g.dinv[d];
    double fu = floor(u);
    if (__double_as_longlong(fu) >= __double_as_longlong(g.top[d])) {  // fu >= n - 2 >= 0, or NaN
        if (x > g.b[d]) *outside = true;
        fu = g.top[d];
    }
    *t = u - fu;
    const unsigned long long k = (unsigned long long)__double_as_longlong(fu);
    const int sh = 1075 - (int)((k >> 52) & 0x7ff);  // fu = m 2^-sh, m its 53-bit significand
    const unsigned long long m = (k & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const int i = sh > 52 ? 0 : (int)(m >> (sh & 63));
    return min(max(i, 0), g.n[d] - 2);
}

// x < a by dx = x - a, whose sign is exact: a negative number, not -0, not NaN
__device__ __forceinline__ bool negative64(double dx)
{
    return (unsigned long long)__double_as_longlong(dx) - 0x8000000000000001ull <
           0x7ff0000000000000ull;
}

// One stencil row: w[0] r0 + w[1] r1 + w[2] r2 + w[3] r3 of both components,
// every product and sum rounded as the reference rounds it.  FIT: the products
// on the integer pipe (intfp64.h, the same bits).
template <bool FIT>
__device__ __forceinline__ double2 row_dot64(const double* w, double2 r0, double2 r1, double2 r2,
                                             double2 r3)
{
    auto mul = [](double a, double b) { return FIT ? ip_mul_fit(a, b) : a * b; };
    return make_double2(mul(w[0], r0.x) + mul(w[1], r1.x) + mul(w[2], r2.x) + mul(w[3], r3.x),
                        mul(w[0], r0.y) + mul(w[1], r1.y) + mul(w[2], r2.y) + mul(w[3], r3.y));
}

// every one of four doubles is in the range of the integer products
__device__ __forceinline__ bool fit4(double a, double b, double c, double d)
{
    return ((((unsigned)__double2hiint(a) - 0x30000000u) |
             ((unsigned)__double2hiint(b) - 0x30000000u) |
             ((unsigned)__double2hiint(c) - 0x30000000u) |
             ((unsigned)__double2hiint(d) - 0x30000000u)) & 0x60000000u) == 0;
}

// the first term of a sum that starts at 0 (one rounding, the product's), and a
// further one
__device__ __forceinline__ double first64(double w, double b)
{
    return ip_fits(ip_bits(w), ip_bits(b)) ? ip_mul_fit(w, b) : __fma_rn(w, b, 0.0);
}
__device__ __forceinline__ double next64(double s, double w, double b) { return s + ip_mul(w, b); }

// sum_a w0[a] sum_b w1[b] sum_c w2[c] C[it+a, ix+b, iy+c] of the interleaved
// (u, v) coefficient block.  The 168 products of a point went to the FP64 pipe
// beside its 126 sums, at 19 cycles of the SM each; on the integer pipe they
// take 11.  Rows or weights out of the integer arithmetic's range (zeros above
// all: velocity masked over land, a point on a grid node) take the FP64 pipe.
// The time levels are a rolled loop: unrolled, the sixteen rows of integer code
// outgrow the instruction caches.
__device__ __forceinline__ void spline_sum_uv64(const SplineGrid& g, const double2* __restrict__ c,
                                                int it, int ix, int iy, const double* w0,
                                                const double* w1, const double* w2, double* u,
                                                double* v)
{
    const bool wfit = fit4(w2[0], w2[1], w2[2], w2[3]);
    double au = 0.0, av = 0.0;
#pragma unroll 1
    for (int a = 0; a < 4; ++a) {
        double su, sv;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const size_t e = (size_t)(it + a) * g.st + (size_t)(ix + b) * g.sx + iy;
            const double2* row = c + e;
            double2 r0 = make_double2(0.0, 0.0), r1 = r0, r2 = r0, r3 = r0;
            if (NBCS_CHECKED(e + 3 < (size_t)g.st * (size_t)(g.n[0] + 2),
                             NBCS_CHECK_SPLINE_GATHER)) {
                r0 = __ldg(row);
                r1 = __ldg(row + 1);
                r2 = __ldg(row + 2);
                r3 = __ldg(row + 3);
            }
            const bool fit = wfit && fit4(r0.x, r1.x, r2.x, r3.x) && fit4(r0.y, r1.y, r2.y, r3.y);
            const double2 d = fit ? row_dot64<true>(w2, r0, r1, r2, r3)
                                  : row_dot64<false>(w2, r0, r1, r2, r3);
            su = b == 0 ? first64(w1[0], d.x) : next64(su, w1[b], d.x);
            sv = b == 0 ? first64(w1[0], d.y) : next64(sv, w1[b], d.y);
        }
        const double wa = a == 0 ? w0[0] : a == 1 ? w0[1] : a == 2 ? w0[2] : w0[3];
        au = a == 0 ? first64(wa, su) : next64(au, wa, su);
        av = a == 0 ? first64(wa, sv) : next64(av, wa, sv);
    }
    *u = au;
    *v = av;
}

// Tricubic evaluation of (u, v) at (t, x, y) with extrapolation mode XM, the
// extrap_mode of the interpolation package's eval_spline that the reference
// passes through (flows.py:121):
//   0 "constant": 0 strictly outside the grid box;
//   1 "nearest":  each coordinate clamped into its axis' [a, b];
//   2 "linear":   the value at the clamped point plus, for each clamped axis
//                 (t, x, y in that order), the derivative along that axis at
//                 the clamped point times the distance beyond the box.
template <int XM>
__device__ __forceinline__ void spline_eval_uv64(const SplineGrid& g, const double2* __restrict__ c,
                                                 double t, double x, double y, double* u,
                                                 double* v)
{
    const double vv[3] = {t, x, y};
    double dl[3], f[3], w[3][4];
    int i[3];
    bool out = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        double cl = vv[d];
        if (XM != 0) cl = vv[d] < g.a[d] ? g.a[d] : (vv[d] > g.b[d] ? g.b[d] : vv[d]);
        const double dx = cl - g.a[d];
        if (XM != 0) dl[d] = vv[d] - cl;
        else if (negative64(dx)) out = true;
        i[d] = spline_locate64(g, d, cl, dx, &f[d], &out);
    }
    if (XM == 0 && out) {
        *u = 0.0;
        *v = 0.0;
        return;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) bspline_w64(f[d], w[d]);
    double au, av;
    spline_sum_uv64(g, c, i[0], i[1], i[2], w[0], w[1], w[2], &au, &av);
    if (XM == 2) {
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            if (dl[d] == 0.0 || isnan(dl[d])) continue;
            double dw[4], gu, gv;
            bspline_dw64(f[d], dw);
            spline_sum_uv64(g, c, i[0], i[1], i[2], d == 0 ? dw : w[0], d == 1 ? dw : w[1],
                            d == 2 ? dw : w[2], &gu, &gv);
            const double s = dl[d] * g.dinv[d];
            au = au + s * gu;
            av = av + s * gv;
        }
    }
    *u = au;
    *v = av;
}

// XM: extrapolation mode (0 constant, 1 nearest, 2 linear)
template <int SPH, int XM = 0>
struct FlowSpline64 {
    SplineGrid g;
    const double2* __restrict__ c;
    double r;

    __device__ __forceinline__ void operator()(double t, const double* y, double* dy,
                                               const Params& P) const
    {
        const double* p = P.v;
        double tt = p[0] * t;
        double u, v;
        if (SPH == 1 || SPH == 2) {
            double xx = SPH == 1 ? py_mod360(y[0] - 180.0) - 180.0 : py_mod360(y[0]);
            double yy = y[1];
            spline_eval_uv64<XM>(g, c, tt, xx, yy, &u, &v);
            dy[0] = p[0] * u * 180.0 / (NBCS_PI * r * nbcs_cos_deg(yy));
            dy[1] = p[0] * v * 180.0 / (NBCS_PI * r);
        } else {
            spline_eval_uv64<XM>(g, c, tt, y[0], y[1], &u, &v);
            dy[0] = p[0] * u;
            dy[1] = p[0] * v;
        }
    }
};

}  // namespace nbcs
