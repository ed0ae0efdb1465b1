// Cauchy-Green / FTLE stencil kernels.
//
//   ftle_grid_2D   diagnostics.py:21-65 (+ utils.gradF_stencil_2D :41-44,
//                  utils.eigvalsh_max_2D :185-189)
//   C_eig_2D       diagnostics.py:200-244
//   ftle_from_eig  diagnostics.py:247-269
//
// One thread per grid point; the flow map is read as double2 (16 B per point)
// and each thread's four neighbours come from the same or adjacent rows, which
// the L1/L2 caches serve, so DRAM sees ~16 B read + 8 B (FTLE) or +16 B
// (eigenvector) written per point.
//
// The arithmetic is the reference's, operation for operation, and what bounds
// it is its FP64 operations: 19 cycles of the SM for an add or a multiply of a
// warp, 137 for a division, 143 for a square root, 570 for log(), against
// some 35 cycles of HBM time for a warp's points.  So the products, quotients,
// roots and logarithms run on the integer pipe (intfp64.h: correctly rounded,
// the same bits; about 13, 17, 27 and 53 cycles) and only the sums, which an
// integer pipe does not do faster, stay on the FP64 pipe beside it (and a pair
// of products, to even out the two pipes).  Kernel times with everything on the
// FP64 pipe and as it is: ftle_kernel 401 x 201 23.5 -> 7.9 us, ceig_kernel 1351
// x 501 with a mask 157 -> 33.6 us, ftle_from_eig_kernel of its eigenvalues 54
// -> 10 us, ftle_evec_kernel 4001 x 4001 1.87 -> 0.36 ms.  The last, whose
// roundings are its own, takes fixed point for the tensor's diagonal and what
// follows (eig2_fixed.h; 10 FP64 operations a point); with 14 FP64 sums a point
// beside integer products it took 0.44 ms (98 % of the FP64 pipe's slots).
// Compiled with -fmad=false.
#include "batch_common.cuh"
#include "eig2_fixed.h"
#include "intfp64.h"
#include "nbcs_internal.cuh"

namespace nbcs {

constexpr int kStencilThreads = 128;

__device__ __forceinline__ bool interior(long k, int nx, const FastDiv& ny, int b = 1)
{
    int i, j;
    row_col(k, ny, &i, &j);
    return i >= b && i < nx - b && j >= b && j < (int)ny.d - b;
}

// The arithmetic of a point, FIT when its differences and the grid spacing are
// ordinary (ordinary_diffs, ordinary_spacing): then every product, quotient and
// root below has operands that fit by themselves or is zero-tested, and the
// range tests of the general form (a few cycles an operation) fall away.
template <bool FIT>
struct Arith {
    static __device__ __forceinline__ double mul(double a, double b)
    {
        return FIT ? ip_mul_fit(a, b) : ip_mul(a, b);
    }
    // a^2, a may be zero
    static __device__ __forceinline__ double sqr(double a)
    {
        return FIT ? ip_sqr_or_zero(a) : ip_mul(a, a);
    }
    static __device__ __forceinline__ double div(double a, const ip_divisor& d)
    {
        return FIT ? ip_div_fit(a, d) : ip_div(a, d);
    }
    // a / d, a may be zero
    static __device__ __forceinline__ double div0(double a, const ip_divisor& d)
    {
        return FIT ? (ip_zero(a) ? a : ip_div_fit(a, d)) : ip_div(a, d);
    }
    // a 2^k, a may be zero
    static __device__ __forceinline__ double scale(double a, int k)
    {
        return FIT ? (ip_zero(a) ? a : ip_scale_fit(a, k)) : ip_scale(a, k);
    }
    // sqrt(a) of a sum of squares
    static __device__ __forceinline__ double root(double a)
    {
        return FIT ? (ip_zero(a) ? a : ip_sqrt_fit(a)) : ip_sqrt(a);
    }
};

// Differences in [2^-63, 2^65) and a spacing in [2^-32, 2^31): gradients in
// [2^-95, 2^96], the tensor's entries below 2^194 and, where a sum of theirs
// cancels without being zero, above 2^-244, their squares in the normal range.
__device__ __forceinline__ bool ordinary_diffs(double2 p, double2 q)
{
    return ((((uint32_t)__double2hiint(p.x) - 0x3c000000u) |
             ((uint32_t)__double2hiint(p.y) - 0x3c000000u) |
             ((uint32_t)__double2hiint(q.x) - 0x3c000000u) |
             ((uint32_t)__double2hiint(q.y) - 0x3c000000u)) & 0x78000000u) == 0;
}

static bool ordinary_spacing(double dx, double dy)
{
    return fabs(dx) >= 0x1p-32 && fabs(dx) < 0x1p31 && fabs(dy) >= 0x1p-32 && fabs(dy) < 0x1p31;
}

// differences across a point: along x and along y of the flow map (x, y)
struct Diffs {
    double2 i, j;
};

__device__ __forceinline__ Diffs diffs_of(double2 ip, double2 im, double2 jp, double2 jm)
{
    return {make_double2(ip.x - im.x, ip.y - im.y), make_double2(jp.x - jm.x, jp.y - jm.y)};
}

__device__ __forceinline__ Diffs diffs_at(const double2* __restrict__ F, long k, int ny)
{
    // interior points only: k - ny >= 0 and k + ny < nx * ny by the caller's test
    return diffs_of(__ldg(F + k + ny), __ldg(F + k - ny), __ldg(F + k + 1), __ldg(F + k - 1));
}

// the whole warp takes the general form when one of its points needs it: two
// forms one after the other would cost more than the slower one (only where the
// two give the same bits: a result must not depend on a point's neighbours)
__device__ __forceinline__ bool all_ordinary(const Diffs& d, bool spacing)
{
    return __all_sync(__activemask(), spacing && ordinary_diffs(d.i, d.j));
}

// Cauchy-Green tensor [[a, b], [b, d]]; dx2, dy2 are the divisors 2 dx, 2 dy
template <bool FIT>
__device__ __forceinline__ void tensor_of(const Diffs& D, const ip_divisor& dx2,
                                          const ip_divisor& dy2, double* a, double* b, double* d)
{
    using A = Arith<FIT>;
    const double dxdx = A::div(D.i.x, dx2), dxdy = A::div(D.j.x, dy2);
    const double dydx = A::div(D.i.y, dx2), dydy = A::div(D.j.y, dy2);
    // b's products on the FP64 pipe even the two pipes out: ftle_kernel 2001 x
    // 1501 90 -> 86 us, with a's too 92
    *b = dxdx * dxdy + dydx * dydy;
    *a = A::mul(dxdx, dxdx) + A::mul(dydx, dydx);
    *d = A::mul(dxdy, dxdy) + A::mul(dydy, dydy);
}

// sqrt((a - d)^2 + 4 b^2)
template <bool FIT>
__device__ __forceinline__ double discriminant(double a, double b, double d)
{
    using A = Arith<FIT>;
    return A::root(A::sqr(a - d) + A::scale(A::sqr(b), 2));
}

// a >= d for the tensor's diagonal (sums of squares: nonnegative or NaN, and
// the reference's comparison is false for NaN)
__device__ __forceinline__ bool diag_ge(double a, double d)
{
    return ip_bits(a) >= ip_bits(d) && ip_bits(a) <= 0x7ff0000000000000ull;
}

// sign of a unit vector: ex >= 0, and ey > 0 where ex is zero
__device__ __forceinline__ void positive_x(double* ex, double* ey)
{
    const long long x = (long long)ip_bits(*ex), y = (long long)ip_bits(*ey);
    if (ip_zero(*ex) ? y < 0 : x < 0) {
        *ex = ip_neg(*ex);
        *ey = ip_neg(*ey);
    }
}

// Symmetric 2x2 eigen-decomposition [[a, b], [b, d]]: the larger eigenvalue by
// the eigvalsh_max_2D closed form, the smaller one in LAPACK dlaev2's
// cancellation-free product form, the unit eigenvector of the larger one from
// the better-conditioned of its two expressions, sign normalised to ex >= 0.
template <bool FIT>
__device__ __forceinline__ void sym2_eig(double a, double b, double d, double* lmin, double* lmax,
                                         double* vx, double* vy)
{
    using A = Arith<FIT>;
    const double tr = a + d, disc = discriminant<FIT>(a, b, d);
    const double l1 = A::scale(tr + disc, -1);
    const bool age = diag_ge(a, d);
    const double acmx = ip_less(d, a) ? a : d, acmn = ip_less(d, a) ? d : a;
    const ip_divisor rl = ip_reciprocal(l1);
    const double l2 = !ip_zero(l1)
                          ? A::div(acmx, rl) * acmn - A::div0(b, rl) * b
                          : 0.5 * (tr - disc);
    double ex = age ? 1.0 : 0.0, ey = age ? 0.0 : 1.0;
    if (!ip_zero(b)) {
        const double e = l1 - (age ? d : a);
        ex = age ? e : b;
        ey = age ? b : e;
        const ip_divisor rn = ip_reciprocal(A::root(A::sqr(ex) + A::sqr(ey)));
        ex = A::div0(ex, rn);
        ey = A::div0(ey, rn);
        positive_x(&ex, &ey);
    }
    *lmin = l2;
    *lmax = l1;
    *vx = ex;
    *vy = ey;
}

// log(l) for the larger eigenvalue l (l > 1)
__device__ __forceinline__ bool stretches(double l)
{
    const unsigned long long u = ip_bits(l);
    return u > 0x3ff0000000000000ull && u <= 0x7ff0000000000000ull;
}

template <bool FIT>
__device__ __forceinline__ double eigmax(const Diffs& D, const ip_divisor& dx2,
                                         const ip_divisor& dy2)
{
    double a, b, d;
    tensor_of<FIT>(D, dx2, dy2, &a, &b, &d);
    return Arith<FIT>::scale((a + d) + discriminant<FIT>(a, b, d), -1);
}

__global__ void __launch_bounds__(kStencilThreads)
ftle_kernel(const double2* __restrict__ F, int nx, FastDiv ny, double scaling, ip_divisor dx2,
            ip_divisor dy2, bool spacing, const uint8_t* __restrict__ mask,
            double* __restrict__ ftle)
{
    const long n = (long)nx * ny.d;
    for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (long)gridDim.x * blockDim.x) {
        double out = 0.0;
        if (interior(k, nx, ny) && !(mask && mask[k])) {
            const Diffs D = diffs_at(F, k, ny.d);
            const double lmax = all_ordinary(D, spacing) ? eigmax<true>(D, dx2, dy2)
                                                         : eigmax<false>(D, dx2, dy2);
            if (stretches(lmax)) out = ip_mul(scaling, ip_log(lmax));
        }
        ftle[k] = out;
    }
}

template <bool FIT>
__device__ __forceinline__ void eig_of(const Diffs& D, const ip_divisor& dx2,
                                       const ip_divisor& dy2, double* l0, double* l1, double* vx,
                                       double* vy)
{
    double a, b, d;
    tensor_of<FIT>(D, dx2, dy2, &a, &b, &d);
    sym2_eig<FIT>(a, b, d, l0, l1, vx, vy);
}

__global__ void __launch_bounds__(kStencilThreads)
ceig_kernel(const double2* __restrict__ F, int nx, FastDiv ny, ip_divisor dx2, ip_divisor dy2,
            bool spacing, const uint8_t* __restrict__ mask, double2* __restrict__ evals,
            double2* __restrict__ evecs)
{
    const long n = (long)nx * ny.d;
    for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (long)gridDim.x * blockDim.x) {
        double2 ev = make_double2(0.0, 0.0);
        double2 v0 = make_double2(0.0, 0.0), v1 = make_double2(0.0, 0.0);
        if (interior(k, nx, ny) && !(mask && mask[k])) {
            double l0, l1, vx, vy;
            const Diffs D = diffs_at(F, k, ny.d);
            if (all_ordinary(D, spacing)) eig_of<true>(D, dx2, dy2, &l0, &l1, &vx, &vy);
            else eig_of<false>(D, dx2, dy2, &l0, &l1, &vx, &vy);
            ev = make_double2(l0, l1);
            v0 = make_double2(ip_neg(vy), vx);  // row 0: columns v_min, v_max
            v1 = make_double2(vx, vy);   // row 1
        }
        evals[k] = ev;
        evecs[2 * k] = v0;
        evecs[2 * k + 1] = v1;
    }
}

// C_tensor_2D (diagnostics.py:69-111) with utils.gradF_aux_stencil_2D
// (:50-84): C11, C12, C22 of the tensor of the +-h particles (the first four
// of the na per point) for 2 <= i < nx-2, 2 <= j < ny-2 unless masked, 0
// elsewhere -- the stencil of ceig_aux_kernel without the eigen-solve.
__global__ void __launch_bounds__(kStencilThreads)
ctensor_aux_kernel(const double2* __restrict__ F, int nx, FastDiv ny, int na, ip_divisor h2,
                   const uint8_t* __restrict__ mask, double* __restrict__ C)
{
    const long n = (long)nx * ny.d;
    for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (long)gridDim.x * blockDim.x) {
        double c11 = 0.0, c12 = 0.0, c22 = 0.0;
        if (interior(k, nx, ny, 2) && !(mask && mask[k])) {
            const double2* A = F + k * na;
            tensor_of<false>(diffs_of(A[0], A[1], A[2], A[3]), h2, h2, &c11, &c12, &c22);
        }
        C[3 * k] = c11;
        C[3 * k + 1] = c12;
        C[3 * k + 2] = c22;
    }
}

// C_eig_aux_2D (diagnostics.py:113-197) with utils.gradF_aux_stencil_2D
// (:50-84) and gradF_main_stencil_2D (:88-124): F is (nx, ny, na, 2).
// eig_main (na = 5): eigenvectors from the aux-particle tensor, eigenvalues
// from the main-grid tensor of the centre particles, for 2 <= i < nx-2,
// 2 <= j < ny-2; otherwise (na = 4) both from the aux tensor, 1-wide border.
__global__ void __launch_bounds__(kStencilThreads)
ceig_aux_kernel(const double2* __restrict__ F, int nx, FastDiv ny, int eig_main, ip_divisor dx2,
                ip_divisor dy2, ip_divisor h2, const uint8_t* __restrict__ mask,
                double2* __restrict__ evals, double2* __restrict__ evecs)
{
    const long n = (long)nx * ny.d;
    const int na = eig_main ? 5 : 4, b = eig_main ? 2 : 1;
    for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (long)gridDim.x * blockDim.x) {
        double2 ev = make_double2(0.0, 0.0);
        double2 v0 = make_double2(0.0, 0.0), v1 = make_double2(0.0, 0.0);
        if (interior(k, nx, ny, b) && !(mask && mask[k])) {
            const double2* A = F + k * na;
            double l0, l1, vx, vy;
            eig_of<false>(diffs_of(A[0], A[1], A[2], A[3]), h2, h2, &l0, &l1, &vx, &vy);
            if (eig_main) {
                double wx, wy;
                eig_of<false>(diffs_of(F[(k + ny.d) * na + 4], F[(k - ny.d) * na + 4],
                                       F[(k + 1) * na + 4], F[(k - 1) * na + 4]),
                              dx2, dy2, &l0, &l1, &wx, &wy);
            }
            ev = make_double2(l0, l1);
            v0 = make_double2(ip_neg(vy), vx);
            v1 = make_double2(vx, vy);
        }
        evals[k] = ev;
        evecs[2 * k] = v0;
        evecs[2 * k + 1] = v1;
    }
}

// whether the reciprocals 1 / (2 dx), 1 / (2 dy) of the spacing are in [2^-31, 2^33)
// (gradients of ordinary differences then in [2^-94, 2^98)): the fused entry
// point and the fields of a batch ask the same of the same numbers
__host__ __device__ __forceinline__ bool ordinary_recips(double rdx, double rdy)
{
    return ((((uint32_t)(ip_bits(rdx) >> 32) - 0x3e000000u) |
             ((uint32_t)(ip_bits(rdy) >> 32) - 0x3e000000u)) & 0x7c000000u) == 0;
}

// FTLE and eigvec_max of one point for the fused ftle_evec_2D entry point: the
// stencil, tensor and larger eigenvalue of ftle_grid_2D / C_eig_2D, with the
// divisions that only scale -- the central differences' 1 / (2 dx), 1 / (2 dy)
// and the FTLE's 1 / (2 |T|) -- taken as products with reciprocals computed
// once on the host.  The smaller eigenvalue, which this entry point does not
// return, is not formed.  The log of the FTLE takes its mantissa part on the
// FP32 pipe: within ~3e-7 relative of ftle_from_eig's where lambda_max >
// 1 + 1e-6.
//
// Ordinary differences (eig2_max_fixed) take 64-bit fixed point from the tensor's
// diagonal on; its off-diagonal entry, which the vector's smaller component is a
// multiple of, is the FP64 one in both forms.
__device__ __forceinline__ double eigvec_max(const Diffs& D, double rdx, double rdy, double* vx,
                                             double* vy)
{
    using A = Arith<false>;
    const double dxdx = A::mul(D.i.x, rdx), dxdy = A::mul(D.j.x, rdy);
    const double dydx = A::mul(D.i.y, rdx), dydy = A::mul(D.j.y, rdy);
    const double b = A::mul(dxdx, dxdy) + A::mul(dydx, dydy);
    const double a = A::mul(dxdx, dxdx) + A::mul(dydx, dydx);
    const double d = A::mul(dxdy, dxdy) + A::mul(dydy, dydy);
    const double l1 = A::scale((a + d) + discriminant<false>(a, b, d), -1);
    const bool age = diag_ge(a, d);
    double ex = age ? 1.0 : 0.0, ey = age ? 0.0 : 1.0;
    if (!ip_zero(b)) {
        const double e = l1 - (age ? d : a);
        ex = age ? e : b;
        ey = age ? b : e;
        const double r = rsqrt(A::mul(ex, ex) + A::mul(ey, ey));
        ex *= r;
        ey *= r;
        positive_x(&ex, &ey);
    }
    *vx = ex;
    *vy = ey;
    return l1;
}

// The same of ordinary differences.  Three of the gradients' scalings and b's
// products on the FP64 pipe beside the integer pipe even the two out: 4001 x 4001
// 363 us, with all four of them there 382, two 365, none (b's products there)
// 389, none at all 426.
__device__ __forceinline__ bool eigvec_max_fit(const Diffs& D, double rdx, double rdy, double* l1,
                                               double* vx, double* vy)
{
    const double dxdx = D.i.x * rdx, dxdy = D.j.x * rdy, dydx = D.i.y * rdx;
    const double dydy = ip_mul_fit(D.j.y, rdy);
    const double b = dxdx * dxdy + dydx * dydy;
    return eig2_max_fixed(dxdx, dxdy, dydx, dydy, b, l1, vx, vy);
}

// FTLE = log(lambda) / (2|T|) to ~3e-7 relative (the contract is 1e-5):
// lambda = 2^e m with m in [1, 2), log(lambda) = e ln 2 + log1p(m - 1); m - 1
// exact, its log1p on the FP32 pipe, the sum in 64-bit fixed point
__device__ __forceinline__ double ftle_of(double l1, double rden)
{
    if (!stretches(l1)) return 0.0;
    const unsigned long long u = ip_bits(l1);
    const int e = (int)(u >> 52) - 1023;
    if (e == 1024) return l1 * rden;  // +inf
    // m - 1 in units of 2^-48, the bits below in the last one: 24 + 24 bits make
    // it a float with one rounding (a 64-bit conversion issues on the FP64 pipe)
    const unsigned top = (unsigned)(u >> 28) & 0xffffffu;
    const unsigned rest = ((unsigned)(u >> 4) & 0xffffffu) | (((unsigned)u & 15u) ? 1u : 0u);
    const float lm =
        log1pf(fmaf((float)top, 16777216.0f, (float)rest) * 3.552713678800501e-15f);
    double l;
    const unsigned lb = __float_as_uint(lm);
    if (e == 0) {  // lm as a double
        l = lb ? ip_double(((unsigned long long)lb << 29) + (896ull << 52)) : 0.0;
    } else {
        // units of 2^-54 (e ln 2 < 710 < 2^10); lm = m24 2^(exponent - 150)
        const int sh = (int)(lb >> 23) - 96;
        const unsigned long long m24 = (lb & 0x7fffffu) | 0x800000u;
        unsigned long long t = (unsigned long long)e * 0x002c5c85fdf473deull;
        t += sh >= 0 ? m24 << sh : (sh > -32 ? m24 >> -sh : 0ull);
        const int z = __clzll((long long)t);
        t <<= z;
        if (ip_fits(ip_bits(rden))) {  // 1 / (2 |T|) is not negative
            const ip_u64 q = ip_high_product(t, ip_left(ip_bits(rden)));
            const int up = (int)(q >> 63);
            return ip_pack(0, ((q >> (9 + up)) + 1) >> 1, ip_exponent(ip_bits(rden)) + 9 - z + up);
        }
        l = ip_pack(0, (t >> 11) + ((t >> 10) & 1), 1023 + 9 - z);
    }
    return ip_mul(l, rden);
}

__device__ __forceinline__ void ftle_evec_point(const double2* __restrict__ F, long k, int ny,
                                                double rdx, double rdy, double rden, bool spacing,
                                                double* f, double2* v)
{
    const Diffs D = diffs_at(F, k, ny);
    // by the point's own differences (the two forms' last bits differ, and a point
    // has the same result in any row block and any batch)
    double l1;
    if (!(spacing && ordinary_diffs(D.i, D.j)) ||
        !eigvec_max_fit(D, rdx, rdy, &l1, &v->x, &v->y))
        l1 = eigvec_max(D, rdx, rdy, &v->x, &v->y);
    *f = ftle_of(l1, rden);
}

__global__ void __launch_bounds__(kStencilThreads)
ftle_evec_kernel(const double2* __restrict__ F, int nx, FastDiv ny, double rden, double rdx,
                 double rdy, bool spacing, const uint8_t* __restrict__ mask,
                 double* __restrict__ ftle, double2* __restrict__ evec)
{
    const long n = (long)nx * ny.d;
    for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (long)gridDim.x * blockDim.x) {
        double f = 0.0;
        double2 v = make_double2(0.0, 0.0);
        if (interior(k, nx, ny) && !(mask && mask[k]))
            ftle_evec_point(F, k, ny.d, rdx, rdy, rden, spacing, &f, &v);
        ftle[k] = f;
        evec[k] = v;
    }
}

__global__ void __launch_bounds__(kStencilThreads)
ftle_from_eig_kernel(const double* __restrict__ ev, long n, long stride, ip_divisor den,
                     double* __restrict__ ftle)
{
    for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (long)gridDim.x * blockDim.x) {
        const double e = ev[k * stride];
        double out = 0.0;
        if (!(ip_bits(e) >> 63) && stretches(e)) out = ip_div(ip_log(e), den);
        ftle[k] = out;
    }
}

// FTLE + eigvec_max of every field of a batch (fields without FTLE own no
// blocks); one 256-thread block per 256-point unit of a field.
__global__ void __launch_bounds__(kFtleBlock)
ftle_batch_kernel(const DevField* __restrict__ fields, int nfields, long long total_blocks)
{
    for (long long b = blockIdx.x; b < total_blocks; b += gridDim.x) {
        const int f = batch_find<kByFtleBlock>(fields, nfields, b);
        const DevField& F = fields[f];
        const long n = (long)F.nx * F.ny;
        const long k = (long)(b - F.block0) * kFtleBlock + threadIdx.x;
        if (k >= n) continue;
        double fv = 0.0;
        double2 v = make_double2(0.0, 0.0);
        const int i = n <= 0x7fffffffL ? (int)((unsigned)k / (unsigned)F.ny) : (int)(k / F.ny);
        const int j = (int)(k - (long)i * F.ny);
        if (i >= 1 && i < F.nx - 1 && j >= 1 && j < F.ny - 1 && !(F.mask && F.mask[k]))
            ftle_evec_point(reinterpret_cast<const double2*>(F.out), k, F.ny, F.rdx, F.rdy,
                            F.rden, ordinary_recips(F.rdx, F.rdy), &fv, &v);
        F.ftle[k] = fv;
        reinterpret_cast<double2*>(F.evec)[k] = v;
    }
}

int launch_ftle_batch(const DevField* fields, int nfields, long long blocks, cudaStream_t s)
{
    long long g = blocks;
    long long cap = (long long)sm_count() * 32;
    if (g > cap) g = cap;
    ftle_batch_kernel<<<(unsigned)g, kFtleBlock, 0, s>>>(fields, nfields, blocks);
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}

static unsigned grid_for(long n)
{
    long b = (n + kStencilThreads - 1) / kStencilThreads;
    long cap = (long)sm_count() * 64;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (unsigned)b;
}

}  // namespace nbcs

using namespace nbcs;

static int check_fm(const double* fm, int32_t nx, int32_t ny)
{
    if (nx < 0 || ny < 0) return set_error(NBCS_ERR_INVALID, "negative grid size");
    if ((long)nx * ny > 0 && !fm) return set_error(NBCS_ERR_INVALID, "flowmap is NULL");
    if (fm && (reinterpret_cast<uintptr_t>(fm) & 15))
        return set_error(NBCS_ERR_INVALID, "flowmap must be 16-byte aligned");
    return NBCS_OK;
}

extern "C" int nbcs_ftle_grid_2d(const double* flowmap, int32_t nx, int32_t ny, double T,
                                 double dx, double dy, const uint8_t* mask, double* ftle,
                                 void* stream)
{
    NBCS_RANGE();
    int rc = check_fm(flowmap, nx, ny);
    if (rc) return rc;
    long n = (long)nx * ny;
    if (n == 0) return NBCS_OK;
    if (!ftle) return set_error(NBCS_ERR_INVALID, "ftle is NULL");
    double scaling = 1.0 / (2.0 * fabs(T));
    ftle_kernel<<<grid_for(n), kStencilThreads, 0, as_stream(stream)>>>(
        reinterpret_cast<const double2*>(flowmap), nx, fast_div(ny), scaling,
        ip_reciprocal(2.0 * dx), ip_reciprocal(2.0 * dy), ordinary_spacing(dx, dy), mask, ftle);
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}

extern "C" int nbcs_c_eig_2d(const double* flowmap, int32_t nx, int32_t ny, double dx, double dy,
                             const uint8_t* mask, double* evals, double* evecs, void* stream)
{
    NBCS_RANGE();
    int rc = check_fm(flowmap, nx, ny);
    if (rc) return rc;
    long n = (long)nx * ny;
    if (n == 0) return NBCS_OK;
    if (!evals || !evecs || ((reinterpret_cast<uintptr_t>(evecs) | reinterpret_cast<uintptr_t>(evals)) & 15))
        return set_error(NBCS_ERR_INVALID, "evals/evecs NULL or not 16-byte aligned");
    ceig_kernel<<<grid_for(n), kStencilThreads, 0, as_stream(stream)>>>(
        reinterpret_cast<const double2*>(flowmap), nx, fast_div(ny), ip_reciprocal(2.0 * dx),
        ip_reciprocal(2.0 * dy), ordinary_spacing(dx, dy), mask,
        reinterpret_cast<double2*>(evals), reinterpret_cast<double2*>(evecs));
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}

extern "C" int nbcs_c_eig_aux_2d(const double* flowmap_aux, int32_t nx, int32_t ny,
                                 int32_t eig_main, double dx, double dy, double h,
                                 const uint8_t* mask, double* evals, double* evecs, void* stream)
{
    NBCS_RANGE();
    if (nx < 0 || ny < 0) return set_error(NBCS_ERR_INVALID, "c_eig_aux: negative grid size");
    long n = (long)nx * ny;
    if (n == 0) return NBCS_OK;
    if (!flowmap_aux || !evals || !evecs ||
        ((reinterpret_cast<uintptr_t>(flowmap_aux) | reinterpret_cast<uintptr_t>(evals) |
          reinterpret_cast<uintptr_t>(evecs)) & 15))
        return set_error(NBCS_ERR_INVALID, "c_eig_aux: NULL or misaligned array");
    ceig_aux_kernel<<<grid_for(n), kStencilThreads, 0, as_stream(stream)>>>(
        reinterpret_cast<const double2*>(flowmap_aux), nx, fast_div(ny), eig_main ? 1 : 0,
        ip_reciprocal(2.0 * dx), ip_reciprocal(2.0 * dy), ip_reciprocal(2.0 * h), mask,
        reinterpret_cast<double2*>(evals), reinterpret_cast<double2*>(evecs));
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}

extern "C" int nbcs_c_tensor_2d(const double* flowmap_aux, int32_t nx, int32_t ny, int32_t naux,
                                double h, const uint8_t* mask, double* C, void* stream)
{
    NBCS_RANGE();
    if (nx < 0 || ny < 0 || naux < 4)
        return set_error(NBCS_ERR_INVALID, "c_tensor: negative grid size or fewer than 4 aux particles");
    long n = (long)nx * ny;
    if (n == 0) return NBCS_OK;
    if (!flowmap_aux || !C || (reinterpret_cast<uintptr_t>(flowmap_aux) & 15))
        return set_error(NBCS_ERR_INVALID, "c_tensor: NULL or misaligned array");
    ctensor_aux_kernel<<<grid_for(n), kStencilThreads, 0, as_stream(stream)>>>(
        reinterpret_cast<const double2*>(flowmap_aux), nx, fast_div(ny), naux,
        ip_reciprocal(2.0 * h), mask, C);
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}

extern "C" int nbcs_ftle_evec_2d(const double* flowmap, int32_t nx, int32_t ny, double T,
                                 double dx, double dy, const uint8_t* mask, double* ftle,
                                 double* evec_max, void* stream)
{
    NBCS_RANGE();
    int rc = check_fm(flowmap, nx, ny);
    if (rc) return rc;
    long n = (long)nx * ny;
    if (n == 0) return NBCS_OK;
    if (!ftle || !evec_max || (reinterpret_cast<uintptr_t>(evec_max) & 15))
        return set_error(NBCS_ERR_INVALID, "ftle/evec_max NULL or misaligned");
    const double rdx = 1.0 / (2.0 * dx), rdy = 1.0 / (2.0 * dy);
    ftle_evec_kernel<<<grid_for(n), kStencilThreads, 0, as_stream(stream)>>>(
        reinterpret_cast<const double2*>(flowmap), nx, fast_div(ny), 1.0 / (2.0 * fabs(T)), rdx,
        rdy, ordinary_recips(rdx, rdy), mask, ftle, reinterpret_cast<double2*>(evec_max));
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}

extern "C" int nbcs_ftle_from_eig(const double* eigval, int64_t n, int64_t stride, double T,
                                  double* ftle, void* stream)
{
    NBCS_RANGE();
    if (n < 0 || stride < 1) return set_error(NBCS_ERR_INVALID, "ftle_from_eig: bad n/stride");
    if (n == 0) return NBCS_OK;
    if (!eigval || !ftle) return set_error(NBCS_ERR_INVALID, "ftle_from_eig: NULL array");
    ftle_from_eig_kernel<<<grid_for(n), kStencilThreads, 0, as_stream(stream)>>>(
        eigval, n, stride, ip_reciprocal(2.0 * fabs(T)), ftle);
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}
