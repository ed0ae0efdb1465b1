// Cubic B-spline prefilter and coefficient packing.
//
// get_interp_arrays_2D (flows.py:9-46) calls interpolation.splines.prefilter
// with k=3: natural boundary conditions (zero second derivative at both ends),
// n+2 coefficients per axis, applied separably along t, x and y.  Each axis
// is a (1,4,1) tridiagonal solve per grid line; one thread solves one line.
// Compiled with -fmad=false, in the same operation order as the CPU oracle.
//
// What bounds it: the recurrence of a line is serial (its roundings are the
// reference's), so a pass lasts the line's length times an element's latency or
// the SM's share of FP64 work, whichever is longer; the data stays in L2.
//  - The forward-elimination pivots 4 - 1/p settle to a fixed double at the
//    15th: a table in the kernel's parameters.  A block used to divide its way
//    through the whole line's pivots first, on one thread, n x 560 cycles.
//  - Products and the divisions by pivots run on the integer pipe (intfp64.h,
//    the same bits; a division 15 cycles of the SM for 137), which leaves two
//    FP64 sums an element.
//  - Both velocity components go in one launch (twice the lines in flight), the
//    loads of a line run two chunks ahead of its recurrence (one chunk, some
//    2500 cycles, still waited for memory a tenth of the time), and one-warp
//    blocks share the lines out evenly.
//  - The table of pivots is read with constant addresses only: a steady chunk
//    has its pivot in registers, and the out-of-line functions get scalars.
//    With the table's address given away its reads were generic loads, a fifth
//    of a warp's time (57, 82 and 62 us for the three passes below).
//  - The inner elements go in chunks of eight without a branch: whether every
//    operand fitted the integer arithmetic is asked once a chunk, which is
//    redone element by element if not.  A branch per product had the products
//    off the recurrence wait in line with it (twice the time).
//  - Lines along y, whose elements are adjacent in memory, are transposed
//    through shared memory (a warp reads 32 lines in 256-byte runs).
// Both components of a 121 x 217 x 101 block, the passes along t, x and y: 376,
// 585 and 329 us in six launches -> 51, 66 and 60 us in three.  What is left is
// latency: an element takes a 64-cycle FP64 sum after an integer product of
// some 80 cycles, and the x pass has five warps an SM.
#include "intfp64.h"
#include "nbcs_internal.cuh"

namespace nbcs {

struct LineSet {
    long n_outer, n_inner;
    long in_os, in_is, out_os, out_is;  // base offsets per outer / inner index
    long s_in, s_out;                   // element strides along the line
};

// the components of one launch (blockIdx.y)
struct PrefilterIO {
    const double* f[2];
    double* c[2];
};

constexpr int kPivots = 15;  // from here on the pivot repeats
struct Pivots {
    double w[kPivots];       // 1 / piv[k]
    ip_divisor d[kPivots];   // divisor piv[k]
};

static Pivots pivots()
{
    Pivots p;
    double piv = 4.0;
    for (int k = 0; k < kPivots; ++k) {
        p.w[k] = 1.0 / piv;
        p.d[k] = ip_reciprocal(piv);
        // the reciprocal's floor: quotients then lie less than two units (four
        // after normalisation) above the computed ones
        const unsigned __int128 r = ((unsigned __int128)IP_SIGN << 64) / p.d[k].B;
        p.d[k].r = r >> 64 ? ~0ull : (ip_u64)r;
        piv = 4.0 - 1.0 / piv;
    }
    return p;
}

__device__ __forceinline__ int pivot_index(int k) { return min(max(k, 0), kPivots - 1); }

// Forward elimination of element k of m (6 f on the right-hand side), r the
// previous element's and w its pivot's reciprocal; back substitution of element
// k, next the following one.  (Scalars, not the table: the table's address, once
// given away, makes every read of it a load from generic memory.)
__device__ __noinline__ double eliminate1(double w, bool first, bool last, double f, double c0,
                                          double cn1, double r)
{
    double rhs = 6.0 * f;
    if (first) rhs -= c0;
    if (last) rhs -= cn1;
    return first ? rhs : rhs - w * r;
}

__device__ __noinline__ double substitute1(double b, ip_u64 B, ip_u64 rec, bool last, double r,
                                           double next)
{
    const ip_divisor d = {rec, B, b};
    return ip_div(last ? r : r - next, d);
}

__device__ __forceinline__ double eliminate(const Pivots& P, int k, int m, double f, double c0,
                                            double cn1, double r)
{
    return eliminate1(P.w[pivot_index(k - 1)], k == 0, k == m - 1, f, c0, cn1, r);
}

__device__ __forceinline__ double substitute(const Pivots& P, int k, int m, double r, double next)
{
    const ip_divisor& d = P.d[pivot_index(k)];
    return substitute1(d.b, d.B, d.r, k == m - 1, r, next);
}

constexpr int kPfWarp = 32;   // lines per block
constexpr int kPfChunk = 8;   // elements at a time

// x / (a pivot in [2, 4), of reciprocal r and significand B) of an operand that
// fits, r rounded down: the quotient lies in [q, q + 4) of the computed one
__device__ __forceinline__ double pivot_div_fit(double x, ip_u64 r, ip_u64 B)
{
    const ip_u64 u = ip_bits(x);
    const ip_u64 A = ip_left(u);
    ip_u64 q = ip_mulhi(A, r);
    int e = ip_exponent(u) - 1;
    const bool small = !(q >> 63);
    if (small) {
        q <<= 1;
        e -= 1;
    }
    unsigned up = (unsigned)(q >> 10) & 1u;
    if (((unsigned)q & 0x7ffu) - 0x3fcu < 4u)
        up = ip_mulhi((q & ~0x7ffull) | 0x400ull, B) < (small ? A : A >> 1);
    return ip_pack(u, (q >> 11) + up, e);
}

// The pivots of a chunk whose lowest element is k: past the table's end they are
// one pivot, in registers
constexpr int kSteady = kPivots + 1;

// kPfChunk inner elements from k on (none of them the first or the last):
// without branches, so that the products off the recurrence overlap it.  False
// when an operand did not fit the integer arithmetic (r is unchanged then).
template <bool STEADY>
__device__ __forceinline__ bool eliminate_chunk(const Pivots& P, int k, const double* f, double* r,
                                                double* out)
{
    ip_u64 bad = 0;
    double rhs[kPfChunk], w[kPfChunk], rr = *r;
#pragma unroll
    for (int j = 0; j < kPfChunk; ++j) {
        bad |= ip_bits(f[j]) - 0x3000000000000000ull;
        rhs[j] = ip_mul_fit(6.0, f[j]);
        w[j] = P.w[STEADY ? kPivots - 1 : pivot_index(k + j - 1)];
    }
#pragma unroll
    for (int j = 0; j < kPfChunk; ++j) {
        bad |= ip_bits(rr) - 0x3000000000000000ull;
        rr = rhs[j] - ip_mul_fit(w[j], rr);
        out[j] = rr;
    }
    if ((unsigned)(bad >> 32) & 0x60000000u) return false;
    *r = rr;
    return true;
}

// the same of the back substitution, from k downwards
template <bool STEADY>
__device__ __forceinline__ bool substitute_chunk(const Pivots& P, int k, const double* r,
                                                 double* next, double* out)
{
    ip_u64 bad = 0, rec[kPfChunk], B[kPfChunk];
    double v = *next;
#pragma unroll
    for (int j = 0; j < kPfChunk; ++j) {
        const int i = STEADY ? kPivots - 1 : pivot_index(k - j);
        rec[j] = P.d[i].r;
        B[j] = P.d[i].B;
    }
#pragma unroll
    for (int j = 0; j < kPfChunk; ++j) {
        const double x = r[j] - v;
        bad |= ip_bits(x) - 0x3000000000000000ull;
        v = pivot_div_fit(x, rec[j], B[j]);
        out[j] = v;
    }
    if ((unsigned)(bad >> 32) & 0x60000000u) return false;
    *next = v;
    return true;
}

// TILE: lines along the fastest axis -- the block's 32 lines of inputs and
// outputs pass through shared memory, 32 x pitch doubles.  Otherwise a warp's
// lines are adjacent in memory and the eliminated right-hand sides wait in the
// output slots.
template <bool TILE>
__global__ void __launch_bounds__(kPfWarp)
prefilter_lines_kernel(PrefilterIO io, int n, LineSet L, const __grid_constant__ Pivots P,
                       int pitch)
{
    extern __shared__ double sh[];
    const double* __restrict__ f = blockIdx.y ? io.f[1] : io.f[0];
    double* c = blockIdx.y ? io.c[1] : io.c[0];
    const int m = n - 2, lane = threadIdx.x;
    const long lines = L.n_outer * L.n_inner;
    const long l0 = (long)blockIdx.x * kPfWarp, l = l0 + lane;
    const bool live = l < lines;
    const long lc = live ? l : lines - 1, o = lc / L.n_inner, q = lc - o * L.n_inner;
    const double* fl = f + o * L.in_os + q * L.in_is;
    double* cl = c + o * L.out_os + q * L.out_is;
    if (n == 1) {
        if (!live) return;
        const double v = fl[0];
        cl[0] = v;
        cl[L.s_out] = v;
        cl[2 * L.s_out] = v;
        return;
    }
    // in shared memory input element i takes slot i + 1 of its line, where its
    // right-hand side and coefficient follow it
    const int nl = (int)(lines - l0 < kPfWarp ? lines - l0 : kPfWarp);
    if (TILE) {
        // the lines follow one another in memory: one run of nl * n doubles, all
        // of its copies in flight at once; the row of element i by a high product
        // (exact: i * n < 2^32)
        const double* src = f + l0 * n;
        const unsigned inv = 0xffffffffu / (unsigned)n + 1u;
        for (int i = lane; i < nl * n; i += kPfWarp) {
            const unsigned row = __umulhi((unsigned)i, inv), col = (unsigned)i - row * (unsigned)n;
            const unsigned dst = (unsigned)__cvta_generic_to_shared(sh + row * pitch + col + 1);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src + i)
                         : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
    }
    const double* in = TILE ? sh + lane * pitch + 1 : fl;   // input element i at in[i * fs]
    double* out = TILE ? sh + lane * pitch : cl;            // coefficient k at out[k * cs]
    const long fs = TILE ? 1 : L.s_in, cs = TILE ? 1 : L.s_out;
    if (live) {
        const double c0 = in[0], cn1 = in[(long)(n - 1) * fs];
        double r = 0.0;
        // elements 1 .. m - 2 in chunks, the first and the last few one by one
        const int chunks = m > 2 ? (m - 2) / kPfChunk : 0, body = 1 + chunks * kPfChunk;
        if (m > 0) {
            r = eliminate(P, 0, m, in[fs], c0, cn1, r);
            out[2 * cs] = r;
        }
        double buf[kPfChunk], ahead[kPfChunk], after[kPfChunk], res[kPfChunk];
#pragma unroll
        for (int j = 0; j < kPfChunk; ++j) {
            buf[j] = chunks > 0 ? in[(long)(j + 2) * fs] : 0.0;
            ahead[j] = chunks > 1 ? in[(long)(kPfChunk + j + 2) * fs] : 0.0;
        }
        for (int k = 1; k < body; k += kPfChunk) {
            const bool more = k + 2 * kPfChunk < body;
#pragma unroll
            for (int j = 0; j < kPfChunk; ++j)
                after[j] = more ? in[(long)(k + 2 * kPfChunk + j + 1) * fs] : 0.0;
            if (!(k >= kSteady ? eliminate_chunk<true>(P, k, buf, &r, res)
                               : eliminate_chunk<false>(P, k, buf, &r, res))) {
#pragma unroll 1
                for (int j = 0; j < kPfChunk; ++j) {
                    r = eliminate(P, k + j, m, in[(long)(k + j + 1) * fs], c0, cn1, r);
                    out[(long)(k + j + 2) * cs] = r;
                }
            } else {
#pragma unroll
                for (int j = 0; j < kPfChunk; ++j) out[(long)(k + j + 2) * cs] = res[j];
            }
#pragma unroll
            for (int j = 0; j < kPfChunk; ++j) {
                buf[j] = ahead[j];
                ahead[j] = after[j];
            }
        }
#pragma unroll 1
        for (int k = m > 0 ? body : 0; k < m; ++k) {
            r = eliminate(P, k, m, in[(long)(k + 1) * fs], c0, cn1, r);
            out[(long)(k + 2) * cs] = r;
        }
        double next = 0.0, last = cn1;  // the coefficient after, and that of element n - 2
#pragma unroll 1
        for (int k = m - 1; k >= (m > 0 ? body : 0); --k) {
            next = substitute(P, k, m, out[(long)(k + 2) * cs], next);
            out[(long)(k + 2) * cs] = next;
            if (k == m - 1) last = next;
        }
#pragma unroll
        for (int j = 0; j < kPfChunk; ++j) {
            buf[j] = chunks > 0 ? out[(long)(body - 1 - j + 2) * cs] : 0.0;
            ahead[j] = chunks > 1 ? out[(long)(body - 1 - kPfChunk - j + 2) * cs] : 0.0;
        }
        for (int k = body - 1; k >= kPfChunk; k -= kPfChunk) {
            const bool more = k - 2 * kPfChunk >= 1;
#pragma unroll
            for (int j = 0; j < kPfChunk; ++j)
                after[j] = more ? out[(long)(k - 2 * kPfChunk - j + 2) * cs] : 0.0;
            if (!(k - kPfChunk >= kSteady ? substitute_chunk<true>(P, k, buf, &next, res)
                                          : substitute_chunk<false>(P, k, buf, &next, res))) {
#pragma unroll 1
                for (int j = 0; j < kPfChunk; ++j) {
                    next = substitute(P, k - j, m, out[(long)(k - j + 2) * cs], next);
                    out[(long)(k - j + 2) * cs] = next;
                }
            } else {
#pragma unroll
                for (int j = 0; j < kPfChunk; ++j) out[(long)(k - j + 2) * cs] = res[j];
            }
#pragma unroll
            for (int j = 0; j < kPfChunk; ++j) {
                buf[j] = ahead[j];
                ahead[j] = after[j];
            }
        }
        if (m > 0 && body > 0 && m > 1) {
            next = substitute(P, 0, m, out[2 * cs], next);
            out[2 * cs] = next;
        } else if (m == 1) {
            next = last = substitute(P, 0, m, out[2 * cs], 0.0);
            out[2 * cs] = next;
        }
        // on two nodes the neighbours of the ends are each other
        out[0] = 2.0 * c0 - (n > 2 ? next : cn1);
        if (!TILE) {
            out[cs] = c0;
            out[(long)n * cs] = cn1;
        }
        out[(long)(n + 1) * cs] = 2.0 * cn1 - (n > 2 ? last : c0);
    }
    if (TILE) {
        __syncwarp();
        double* dst = c + l0 * (n + 2);
        const unsigned inv = 0xffffffffu / (unsigned)(n + 2) + 1u;
#pragma unroll 8
        for (int i = lane; i < nl * (n + 2); i += kPfWarp) {
            const unsigned row = __umulhi((unsigned)i, inv);
            dst[i] = sh[row * pitch + ((unsigned)i - row * (unsigned)(n + 2))];
        }
    }
}

// FP64 (u, v) per node, and the FP32 "quad" layout: entry k = (u_j, v_j) for
// j = k .. k+3 (32 bytes; zeros past the end) so a 4-tap stencil row is one
// aligned 32-byte load.
// Each thread converts its own node's pair once (an FP64-to-FP32 conversion
// issues on the FP64 pipe, 16 cycles) and takes the three that follow from the
// lanes after it; the last three lanes of a warp only convert.
__global__ void __launch_bounds__(256)
pack_uv_kernel(const double* __restrict__ cu, const double* __restrict__ cv, long n,
               double2* __restrict__ uv, float4* __restrict__ uv32)
{
    const int lane = threadIdx.x & 31;
    constexpr int kNew = 29;  // nodes a warp writes
    const long warps = ((long)gridDim.x * blockDim.x) >> 5;
    for (long w = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * kNew < n; w += warps) {
        const long k = w * kNew + lane;
        double u = 0.0, v = 0.0;
        if (k < n) {
            u = cu[k];
            v = cv[k];
        }
        const float a = (float)u, b = (float)v;
        float q[8] = {a, b};
#pragma unroll
        for (int j = 1; j < 4; ++j) {
            q[2 * j] = __shfl_down_sync(0xffffffffu, a, j);
            q[2 * j + 1] = __shfl_down_sync(0xffffffffu, b, j);
        }
        if (lane < kNew && k < n) {
            uv[k] = make_double2(u, v);
            if (uv32) {
                uv32[2 * k] = make_float4(q[0], q[1], q[2], q[3]);
                uv32[2 * k + 1] = make_float4(q[4], q[5], q[6], q[7]);
            }
        }
    }
}

static const int kMaxLine = 12000;  // longest axis taken

// Shared memory of a block (one warp) up to which lines along y are transposed
// through it; longer ones are read line by line.
constexpr int kPfShared = 96 * 1024;

static int run_pass(const PrefilterIO& io, int count, int n, const LineSet& L, cudaStream_t s)
{
    const long lines = L.n_outer * L.n_inner;
    if (lines == 0) return NBCS_OK;
    const long blocks = (lines + kPfWarp - 1) / kPfWarp;
    if (blocks > 0x7fffffffL) return set_error(NBCS_ERR_UNSUPPORTED, "prefilter: too many lines");
    const dim3 grid((unsigned)blocks, (unsigned)count);
    const Pivots P = pivots();
    const int pitch = (n + 2) | 1;  // odd: the 32 lines' slots fall in different banks
    const size_t tile = sizeof(double) * kPfWarp * (size_t)pitch;
    // contiguous lines, one after the other: the y pass
    const bool rows = L.s_in == 1 && L.s_out == 1 && L.in_is == n && L.out_is == n + 2 &&
                      L.in_os == L.n_inner * L.in_is && L.out_os == L.n_inner * L.out_is;
    if (n > 1 && rows && tile <= (size_t)kPfShared) {
        if (tile > 48 * 1024)
            NBCS_CUDA_TRY(cudaFuncSetAttribute(prefilter_lines_kernel<true>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kPfShared));
        prefilter_lines_kernel<true><<<grid, kPfWarp, tile, s>>>(io, n, L, P, pitch);
    } else {
        prefilter_lines_kernel<false><<<grid, kPfWarp, 0, s>>>(io, n, L, P, 0);
    }
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}

// the three passes of `count` (1 or 2) fields; scratch holds both intermediate
// arrays of each
static int prefilter_fields(const double* const* f, double* const* coef, int count, int32_t nt,
                            int32_t nx, int32_t ny, void* scratch, cudaStream_t s)
{
    const long NT = nt + 2, NX = nx + 2, NY = ny + 2;
    const size_t n1 = (size_t)NT * nx * ny, n2 = (size_t)NT * NX * ny;
    double* tmp = static_cast<double*>(scratch);  // (NT, nx, ny) each
    double* tmp2 = tmp + (size_t)count * n1;      // (NT, NX, ny) each
    PrefilterIO t = {}, x = {}, y = {};
    for (int k = 0; k < count; ++k) {
        t.f[k] = f[k];
        t.c[k] = tmp + (size_t)k * n1;
        x.f[k] = t.c[k];
        x.c[k] = tmp2 + (size_t)k * n2;
        y.f[k] = x.c[k];
        y.c[k] = coef[k];
    }
    const LineSet Lt = {nx, ny, ny, 1, ny, 1, (long)nx * ny, (long)nx * ny};
    const LineSet Lx = {NT, ny, (long)nx * ny, 1, NX * ny, 1, ny, ny};
    const LineSet Ly = {NT, NX, NX * ny, ny, NX * NY, NY, 1, 1};
    int rc = run_pass(t, count, nt, Lt, s);
    if (!rc) rc = run_pass(x, count, nx, Lx, s);
    if (!rc) rc = run_pass(y, count, ny, Ly, s);
    return rc;
}

static int check_prefilter(int32_t nt, int32_t nx, int32_t ny, const void* scratch,
                           size_t scratch_bytes, size_t need)
{
    if (nt > kMaxLine || nx > kMaxLine || ny > kMaxLine)
        return set_error(NBCS_ERR_UNSUPPORTED, "prefilter: axis longer than %d", kMaxLine);
    if (!scratch || scratch_bytes < need)
        return set_error(NBCS_ERR_SCRATCH, "prefilter: scratch needs %zu bytes", need);
    return NBCS_OK;
}

}  // namespace nbcs

using namespace nbcs;

extern "C" size_t nbcs_spline_prefilter_scratch_bytes(int32_t nt, int32_t nx, int32_t ny)
{
    if (nt < 1 || nx < 1 || ny < 1) return 0;
    size_t NT = (size_t)nt + 2, NX = (size_t)nx + 2;
    return sizeof(double) * (NT * nx * ny + NT * NX * ny);
}

extern "C" int nbcs_spline_prefilter_3d(const double* f, int32_t nt, int32_t nx, int32_t ny,
                                        double* coef, void* scratch, size_t scratch_bytes,
                                        void* stream)
{
    NBCS_RANGE();
    if (nt < 1 || nx < 1 || ny < 1 || !f || !coef)
        return set_error(NBCS_ERR_INVALID, "prefilter: bad sizes or NULL arrays");
    int rc = check_prefilter(nt, nx, ny, scratch, scratch_bytes,
                             nbcs_spline_prefilter_scratch_bytes(nt, nx, ny));
    if (rc) return rc;
    return prefilter_fields(&f, &coef, 1, nt, nx, ny, scratch, as_stream(stream));
}

extern "C" int nbcs_spline_prefilter_uv(const double* u, const double* v, int32_t nt, int32_t nx,
                                        int32_t ny, double* coef_u, double* coef_v, void* scratch,
                                        size_t scratch_bytes, void* stream)
{
    NBCS_RANGE();
    if (nt < 1 || nx < 1 || ny < 1 || !u || !v || !coef_u || !coef_v)
        return set_error(NBCS_ERR_INVALID, "prefilter_uv: bad sizes or NULL arrays");
    int rc = check_prefilter(nt, nx, ny, scratch, scratch_bytes,
                             2 * nbcs_spline_prefilter_scratch_bytes(nt, nx, ny));
    if (rc) return rc;
    const double* f[2] = {u, v};
    double* c[2] = {coef_u, coef_v};
    return prefilter_fields(f, c, 2, nt, nx, ny, scratch, as_stream(stream));
}

extern "C" int nbcs_spline_pack_uv(const double* cu, const double* cv, int64_t n, double* coef_uv,
                                   float* coef_uv32, void* stream)
{
    NBCS_RANGE();
    if (n < 0 || (n > 0 && (!cu || !cv || !coef_uv)))
        return set_error(NBCS_ERR_INVALID, "pack_uv: bad arguments");
    if ((reinterpret_cast<uintptr_t>(coef_uv) & 15) || (reinterpret_cast<uintptr_t>(coef_uv32) & 31))
        return set_error(NBCS_ERR_INVALID,
                         "pack_uv: coef_uv must be 16-byte and coef_uv32 32-byte aligned");
    if (n == 0) return NBCS_OK;
    long blocks = (n + 231) / 232;  // eight warps of 29 nodes
    long cap = (long)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    pack_uv_kernel<<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(
        cu, cv, n, reinterpret_cast<double2*>(coef_uv), reinterpret_cast<float4*>(coef_uv32));
    NBCS_LAUNCH_CHECK();
    return NBCS_OK;
}
