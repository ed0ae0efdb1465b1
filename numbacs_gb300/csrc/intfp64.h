/*
 * IEEE double multiplication, division, square root and logarithm on the
 * integer pipe.
 *
 * GB300 executes an FP64 instruction of a warp in 19 cycles of the SM, a
 * division in 137, a square root in 143 and log() in about 570; a 32-bit
 * integer or logic instruction takes half a cycle and the high half of a
 * 64 x 64-bit product 4.3 (all measured).  The operations below work on the
 * 53-bit significands in 64-bit registers: 13 cycles for a product (15 with the
 * test of the operands' ranges), 17 for a quotient whose divisor's reciprocal is
 * at hand, 34 for one with the reciprocal, 27 for a square root, 53 for a
 * logarithm, 115 for a sine and cosine (the library's: 438), and they run beside
 * the FP64 pipe.
 *
 * ip_mul, ip_div and ip_sqrt are correctly rounded (round to nearest even): the
 * same bits as * / sqrt.  The product is exact in 106 bits.  Quotient and root
 * come from a hardware FP32 estimate and two Newton-Raphson corrections in
 * fixed point (64 bits, a few units off); where those units could change the
 * rounding, the midpoint itself is multiplied back and compared.  ip_log is
 * within 0.55 ulp (a table of 128 reciprocals, after P. T. P. Tang's
 * table-driven logarithm, 1990, with log1p of the exact remainder by its
 * Taylor series in fixed point).
 *
 * Operands outside [2^-255, 2^256) in magnitude -- zeros, subnormals,
 * infinities and NaN among them -- take the ordinary FP64 operation.
 *
 * Plain C++ on both sides, so that the host can check every operation against
 * its own FP64 arithmetic.
 */
#ifndef NBCS_INTFP64_H
#define NBCS_INTFP64_H

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define NBCS_IHD __host__ __device__ __forceinline__
#else
#define NBCS_IHD static inline
#endif

typedef unsigned long long ip_u64;

NBCS_IHD ip_u64 ip_bits(double d)
{
#ifdef __CUDA_ARCH__
    return (ip_u64)__double_as_longlong(d);
#else
    ip_u64 u;
    memcpy(&u, &d, sizeof u);
    return u;
#endif
}

NBCS_IHD double ip_double(ip_u64 u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double d;
    memcpy(&d, &u, sizeof d);
    return d;
#endif
}

NBCS_IHD ip_u64 ip_mulhi(ip_u64 a, ip_u64 b)
{
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (ip_u64)(((unsigned __int128)a * b) >> 64);
#endif
}

NBCS_IHD uint32_t ip_mulhi32(uint32_t a, uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((ip_u64)a * b) >> 32);
#endif
}

NBCS_IHD int ip_clz64(ip_u64 a)
{
#ifdef __CUDA_ARCH__
    return __clzll((long long)a);
#else
    return __builtin_clzll(a);
#endif
}

/* FP32 estimate of 1 / f or 1 / sqrt(f) with a relative error below 2^-22, as a
 * 31-bit fixed-point number in [2^30, 2^31) (value times 2^30); fb are the bits
 * of a float f whose result lies in [1, 2] */
NBCS_IHD uint32_t ip_estimate(uint32_t fb, bool root)
{
    float f, y;
    uint32_t yb;
#ifdef __CUDA_ARCH__
    f = __uint_as_float(fb);
    if (root) asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    else asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    yb = __float_as_uint(fminf(fmaxf(y, 1.0f), 1.99999988f));
#else
    memcpy(&f, &fb, sizeof f);
    y = root ? 1.0f / sqrtf(f) : 1.0f / f;
    y = fminf(fmaxf(y, 1.0f), 1.99999988f);
    memcpy(&yb, &y, sizeof yb);
#ifdef NBCS_INTFP64_ESTIMATE_ULPS /* host tests: estimates as far off as the device's may be */
    yb += (uint32_t)NBCS_INTFP64_ESTIMATE_ULPS;
    if (yb < 0x3f800000u) yb = 0x3f800000u;
    if (yb > 0x3fffffffu) yb = 0x3fffffffu;
#endif
#endif
    return ((yb & 0x7fffffu) | 0x800000u) << 7;
}

/* The FP64 pipe's operations where they are the exception (operands out of
 * range, a coordinate in the last cell).  Out of line: in line the compiler
 * issues them under a false predicate beside the usual path, at the FP64 pipe's
 * full price. */
#ifdef __CUDACC__
static __device__ __noinline__ double ip_pipe_mul(double a, double b) { return a * b; }
static __device__ __noinline__ double ip_pipe_sub(double a, double b) { return a - b; }
static __device__ __noinline__ bool ip_pipe_greater(double a, double b) { return a > b; }
#endif
#ifdef __CUDA_ARCH__
#define IP_PIPE_MUL(a, b) ip_pipe_mul(a, b)
#define IP_PIPE_SUB(a, b) ip_pipe_sub(a, b)
#else
#define IP_PIPE_MUL(a, b) ((a) * (b))
#define IP_PIPE_SUB(a, b) ((a) - (b))
#endif

#define IP_IMPLICIT 0x0010000000000000ull
#define IP_FRACTION 0x000fffffffffffffull
#define IP_SIGN 0x8000000000000000ull

/* the exponent of every operand is in [-255, 256): its field in [0x300, 0x4ff] */
NBCS_IHD bool ip_fits(ip_u64 a)
{
    return ((((uint32_t)(a >> 32)) - 0x30000000u) & 0x60000000u) == 0;
}
NBCS_IHD bool ip_fits(ip_u64 a, ip_u64 b)
{
    return (((((uint32_t)(a >> 32)) - 0x30000000u) | (((uint32_t)(b >> 32)) - 0x30000000u)) &
            0x60000000u) == 0;
}
NBCS_IHD int ip_exponent(ip_u64 a) { return (int)((a >> 52) & 0x7ff); }
/* the significand with its top bit at bit 63 */
NBCS_IHD ip_u64 ip_left(ip_u64 a) { return (a << 11) | IP_SIGN; }

/* sign, significand q (53 bits, the top one at bit 52; 2^53 carries into the
 * exponent) and biased exponent e */
NBCS_IHD double ip_pack(ip_u64 sign, ip_u64 q, int e)
{
    return ip_double((sign & IP_SIGN) | (q + ((ip_u64)(uint32_t)(e - 1) << 52)));
}

/* -a without an FP64 instruction */
NBCS_IHD double ip_neg(double a)
{
#ifdef __CUDA_ARCH__
    return __hiloint2double(__double2hiint(a) ^ (int)0x80000000u, __double2loint(a));
#else
    return -a;
#endif
}

/* a < b for operands that are not negative (NaN counts as the largest) */
NBCS_IHD bool ip_less(double a, double b) { return ip_bits(a) < ip_bits(b); }
NBCS_IHD bool ip_zero(double a)
{
#ifdef __CUDA_ARCH__
    /* from the halves: the compiler turns the 64-bit test into an FP64 compare */
    return (((unsigned)__double2hiint(a) << 1) | (unsigned)__double2loint(a)) == 0;
#else
    return (ip_bits(a) << 1) == 0;
#endif
}
/* a 2^k of an operand that fits */
NBCS_IHD double ip_scale_fit(double a, int k)
{
    return ip_double(ip_bits(a) + ((ip_u64)(int64_t)k << 52));
}

/* (P << sh) rounded to its top 53 bits (nearest, ties to even) and packed: P the
 * 128-bit number t3 : mid : low, whose top bit is at 116 - sh; se the sign and
 * the biased exponent less one */
NBCS_IHD double ip_round(ip_u64 t3, uint32_t mid, uint32_t low, uint32_t sh, uint32_t se)
{
#ifdef __CUDA_ARCH__
    const uint32_t h0 = (uint32_t)t3, h1 = (uint32_t)(t3 >> 32);
    const uint32_t m1 = __funnelshift_l(h0, h1, sh), m0 = __funnelshift_l(mid, h0, sh);
    const uint32_t rest = __funnelshift_l(low, mid, sh) | min(low << sh, 1u);
    uint32_t carry, r0, r1;
    asm("add.cc.u32 %0, %3, %4;\n\taddc.cc.u32 %1, %5, 0;\n\taddc.u32 %2, %6, %7;"
        : "=r"(carry), "=r"(r0), "=r"(r1)
        : "r"(rest), "r"(0x7fffffffu + (m0 & 1u)), "r"(m0), "r"(m1), "r"(se));
    (void)carry;
    return __hiloint2double((int)r1, (int)r0);
#else
    const ip_u64 lo = ((ip_u64)mid << 32) | low, rest = lo << sh;
    ip_u64 m = (t3 << sh) | (lo >> (64 - sh));
    m += rest > 0x7fffffffffffffffull + (~m & 1) ? 1 : 0;
    return ip_double(m + ((ip_u64)se << 32));
#endif
}

/* a * b of operands that fit: four 32 x 32-bit products, 106 bits exact */
NBCS_IHD double ip_mul_fit(double a, double b)
{
    const ip_u64 ua = ip_bits(a), ub = ip_bits(b);
    const uint32_t ah = (uint32_t)(ua >> 32), a0 = (uint32_t)ua, bh = (uint32_t)(ub >> 32),
                   b0 = (uint32_t)ub;
    const uint32_t a1 = (ah & 0xfffffu) | 0x100000u, b1 = (bh & 0xfffffu) | 0x100000u;
    const ip_u64 t0 = (ip_u64)a0 * b0;
    const ip_u64 t1 = (ip_u64)a0 * b1 + (t0 >> 32);
    const ip_u64 t2 = (ip_u64)a1 * b0 + (uint32_t)t1;
    const ip_u64 t3 = (ip_u64)a1 * b1 + (t1 >> 32) + (t2 >> 32);
    const uint32_t n = (uint32_t)(t3 >> 41);  /* 1 when the product is 2^105 or more */
    return ip_round(t3, (uint32_t)t2, (uint32_t)t0, 12u - n,
                    (ah & 0xfff00000u) + (bh & 0xfff00000u) + (n << 20) - 0x40000000u);
}

/* the same for operands of which each is zero or fits, the product then +0 */
NBCS_IHD double ip_sqr_or_zero(double a)
{
    return ip_zero(a) ? 0.0 : ip_mul_fit(a, a);
}

/* a * b */
NBCS_IHD double ip_mul(double a, double b)
{
    return ip_fits(ip_bits(a), ip_bits(b)) ? ip_mul_fit(a, b) : IP_PIPE_MUL(a, b);
}

/* a 2^k, exact */
NBCS_IHD double ip_scale(double a, int k)
{
    const ip_u64 u = ip_bits(a);
    return ip_fits(u) ? ip_double(u + ((ip_u64)(int64_t)k << 52))
                      : IP_PIPE_MUL(a, ip_double((ip_u64)(1023 + k) << 52));
}

/* a - b of operands whose exponents are at most nine apart (of which one fits,
 * then: both are far from the ends of the exponent range): the significands'
 * sum or difference is exact in 63 bits, and rounded once */
NBCS_IHD double ip_sub(double a, double b)
{
    const ip_u64 ua = ip_bits(a), ub = ip_bits(b);
    const int ea = ip_exponent(ua), eb = ip_exponent(ub), apart = ea - eb;
    if ((uint32_t)(apart + 9) > 18u || !ip_fits(ua)) return IP_PIPE_SUB(a, b);
    const int sa = 9 + (apart < 0 ? apart : 0), sb = 9 - (apart > 0 ? apart : 0);
    const ip_u64 A = ((ua & IP_FRACTION) | IP_IMPLICIT) << sa;
    const ip_u64 B = ((ub & IP_FRACTION) | IP_IMPLICIT) << sb;
    const ip_u64 opposite = (ip_u64)((int64_t)(ua ^ ub) >> 63);
    const int64_t d = (int64_t)(A - ((B ^ opposite) - opposite));
    const ip_u64 m = (ip_u64)(d < 0 ? -d : d);
    if (!m) return 0.0;
    const int n = ip_clz64(m);
    const ip_u64 L = m << n, q = L >> 11;
    const uint32_t up = ((uint32_t)L & 0x7ffu) + ((uint32_t)q & 1u) > 0x400u ? 1u : 0u;
    return ip_pack(ua ^ (ip_u64)d, q + up, ea + 11 - sa - n);
}

/* A divisor: r = 2^127 / B with the significand B (top bit at 63), to within
 * four units below or above, and b itself for the operands that do not fit. */
struct ip_divisor {
    ip_u64 r, B;
    double b;
};

/* r from the significand B (top bit at 63) and the estimate Y = 2^93 / B */
NBCS_IHD ip_u64 ip_refine(ip_u64 B, uint32_t Y)
{
    /* B Y - 1 in units of 2^-64, below 2^42 */
    const int64_t E = (int64_t)((ip_mulhi(B, Y) << 34) | ((B * Y) >> 30));
    ip_u64 r = ((ip_u64)Y << 33) - (ip_u64)(((int64_t)(int32_t)(E >> 13) * (int32_t)Y) >> 18);
    /* the same of the better estimate, in units of 2^-63 */
    const int32_t E2 = (int32_t)(ip_mulhi(B, r) - IP_SIGN);
    r -= (ip_u64)(((int64_t)E2 * (int32_t)Y) >> 30);
    return r >> 63 ? r : ~0ull;  /* a power of two: 2^64 has wrapped */
}

NBCS_IHD ip_divisor ip_reciprocal(double b)
{
    const ip_u64 ub = ip_bits(b);
    ip_divisor d;
    d.b = b;
    d.B = ip_left(ub);
    d.r = ip_refine(d.B, ip_estimate((126u << 23) | ((uint32_t)(ub >> 29) & 0x7fffffu), false));
    return d;
}

/* a / d.b of operands that fit */
NBCS_IHD double ip_div_fit(double a, const ip_divisor& d)
{
    const ip_u64 ua = ip_bits(a), ub = ip_bits(d.b);
    const ip_u64 A = ip_left(ua);
    ip_u64 q = ip_mulhi(A, d.r);  /* A / B 2^63, five units off at most */
    int e = ip_exponent(ua) - ip_exponent(ub) + 1023;
    const bool small = !(q >> 63);
    if (small) {
        q <<= 1;
        e -= 1;
    }
    uint32_t up = (uint32_t)(q >> 10) & 1u;
    if (((uint32_t)q & 0x7ffu) - (0x400u - 12u) < 24u)
        /* too near the midpoint of two doubles to tell: A / B is above it when
         * midpoint * B is below A at its scale (it is never equal) */
        up = ip_mulhi((q & ~0x7ffull) | 0x400ull, d.B) < (small ? A : A >> 1);
    return ip_pack(ua ^ ub, (q >> 11) + up, e);
}

/* a / d.b */
NBCS_IHD double ip_div(double a, const ip_divisor& d)
{
    const ip_u64 ua = ip_bits(a), ub = ip_bits(d.b);
    if (ip_fits(ua, ub)) return ip_div_fit(a, d);
    if (ip_fits(ub) && ip_zero(a)) return ip_double((ua ^ ub) & IP_SIGN);
    return a / d.b;
}

/* 2^64 sqrt(M / 2^64), three units off at most, of M in [2^62, 2^64) and the
 * estimate Y of its reciprocal root */
NBCS_IHD ip_u64 ip_root64(ip_u64 M, uint32_t Y)
{
    const uint32_t S = (uint32_t)(((ip_u64)(uint32_t)(M >> 32) * Y) >> 31);  /* root 2^31 */
    const int64_t D = (int64_t)(M - (((ip_u64)S * S) << 2));  /* below 2^43 */
    const ip_u64 r =
        ((ip_u64)S << 33) + (ip_u64)(((int64_t)(int32_t)(D >> 13) * (int32_t)Y) >> 18);
    const int32_t D2 = (int32_t)(M - ip_mulhi(r, r));
    return r + (ip_u64)(((int64_t)D2 * (int32_t)Y) >> 31);
}

/* 2^63 / sqrt(M / 2^64), below 2^64, a few units of 2^2 off, of the same */
NBCS_IHD ip_u64 ip_rroot64(ip_u64 M, uint32_t Y)
{
    /* y += y (1 - M y^2) / 2 twice; 1 - M y^2 in units of 2^-62 */
    const int64_t E = (int64_t)(0x4000000000000000ull - ip_mulhi(M, ((ip_u64)Y * Y) << 2));
    const ip_u64 r =
        ((ip_u64)Y << 32) + (ip_u64)(((int64_t)(int32_t)(E >> 12) * (int32_t)Y) >> 19);
    const int32_t E2 = (int32_t)(0x4000000000000000ull - ip_mulhi(M, ip_mulhi(r, r) << 2));
    ip_u64 q = r + (ip_u64)(((int64_t)E2 * (int32_t)Y) >> 31);  /* 2^62 / root, 2^62 to 2^63 */
    if (!(q >> 62)) q = 0x4000000000000000ull;  /* a root just below 1 */
    return q >> 63 ? ~0ull : q << 1;
}

/* the estimate of the reciprocal root of M / 2^64, M in [2^62, 2^64) */
NBCS_IHD uint32_t ip_root_estimate(ip_u64 M)
{
    const uint32_t s = (uint32_t)(M >> 63) ^ 1u, h = (uint32_t)(M >> 32) << s;
    return ip_estimate(((126u - s) << 23) | ((h >> 8) & 0x7fffffu), true);
}

/* sqrt(x) of a positive normal number */
NBCS_IHD double ip_sqrt_fit(double x)
{
    const ip_u64 u = ip_bits(x);
    const int e = ip_exponent(u);
    const uint32_t s = (uint32_t)e & 1u;
    /* M / 2^64 in [1/4, 1), an even power of two from x */
    const ip_u64 M = ((u & IP_FRACTION) | IP_IMPLICIT) << (11 - s);
    const uint32_t Y =
        ip_estimate(((126u - s) << 23) | ((uint32_t)(u >> 29) & 0x7fffffu), true);
    const ip_u64 q = ip_root64(M, Y);
    uint32_t up = (uint32_t)(q >> 10) & 1u;
    if (((uint32_t)q & 0x7ffu) - (0x400u - 6u) < 12u) {
        const ip_u64 mid = (q & ~0x7ffull) | 0x400ull;
        up = ip_mulhi(mid, mid) < M;  /* the root is never a midpoint */
    }
    return ip_pack(0, (q >> 11) + up, (e + 1022 + (int)s) >> 1);
}

/* sqrt(x) */
NBCS_IHD double ip_sqrt(double x)
{
    const ip_u64 u = ip_bits(x);
    return ip_fits(u) && !(u >> 63) ? ip_sqrt_fit(x) : sqrt(x);
}

struct ip_log_entry {
    uint32_t c;   /* 2^10 times a reciprocal of 1 + i / 128, rounded up */
    ip_u64 l;     /* -log(c 2^-10) in units of 2^-64 */
};

#ifdef __CUDACC__
#define IP_TABLE __device__ const
#else
#define IP_TABLE const
#endif
static IP_TABLE ip_log_entry ip_log_table[128] = {
    {1024u, 0x0000000000000000ull}, {1017u, 0x01c189cbb0e27fabull}, {1009u, 0x03c719c606662177ull}, {1001u, 0x05d0c874f401b4a7ull},
    {993u, 0x07dea6c59e0a156dull}, {986u, 0x09ae45fd5098357dull}, {979u, 0x0b8132d2a873bb90ull}, {971u, 0x0d9aeecdac5d5675ull},
    {964u, 0x0f7518e0035c3dd8ull}, {957u, 0x1152b799bb3cc89bull}, {950u, 0x1333d7f8183f4b6aull}, {943u, 0x1518874226130a1eull},
    {937u, 0x16bad83c1883b5e8ull}, {930u, 0x18a6477a91dc28c1ull}, {924u, 0x1a4e7640b1bc37a9ull}, {917u, 0x1c40d6425a5cb112ull},
    {911u, 0x1def0d8d466db8b0ull}, {904u, 0x1fe89139dbd56595ull}, {898u, 0x219cfd9b9985194bull}, {892u, 0x235456fc47ee53c7ull},
    {886u, 0x250ea7782357494eull}, {880u, 0x26cbf9602b202c5full}, {874u, 0x288c573b9367b7a7ull}, {869u, 0x2a0456525ed48a06ull},
    {863u, 0x2bca6628982e31f4ull}, {857u, 0x2d93a0fa407f8e30ull}, {852u, 0x2f131b0a8898e67cull}, {846u, 0x30e2426ea1d328ebull},
    {841u, 0x3266bcbab293115cull}, {835u, 0x343bf881e36fe1f1ull}, {830u, 0x35c594dece57a8d6ull}, {825u, 0x37519215c95a32e8ull},
    {820u, 0x38dff78de01ee139ull}, {815u, 0x3a70ccd0e3e8c9afull}, {810u, 0x3c04198c46b56a80ull}, {805u, 0x3d99e591fd24139cull},
    {800u, 0x3f3238d96766f2fbull}, {795u, 0x40cd1b8041818a00ull}, {790u, 0x426a95cb9b1b50a2ull}, {785u, 0x440ab028d7307021ull},
    {781u, 0x45597bb5157f0c53ull}, {776u, 0x46fe658d69ae5377ull}, {772u, 0x485115b43ae350fcull}, {767u, 0x49faebd63632733cull},
    {763u, 0x4b51980ab733b979ull}, {758u, 0x4d00784abb2e838dull}, {754u, 0x4e5b38d66efd4f8cull}, {749u, 0x500f421b3a9e6ef5ull},
    {745u, 0x516e30285f7c4ddcull}, {741u, 0x52cf01dc99fa692eull}, {737u, 0x5431bc7446e5f195ull}, {733u, 0x55966541a545317full},
    {729u, 0x56fd01ad50f6c7eeull}, {725u, 0x58659736c0b07ba9ull}, {721u, 0x59d02b74c77a51daull}, {717u, 0x5b3cc41619c3b0b2ull},
    {713u, 0x5cab66e1d6318170ull}, {709u, 0x5e1c19b812457d19ull}, {705u, 0x5f8ee2926b00155eull}, {701u, 0x6103c784999fc03cull},
    {698u, 0x621cd960c9f33b8full}, {694u, 0x63957e6cd26e0de2ull}, {690u, 0x651050d280c965c1ull}, {687u, 0x662de0468fb96d4aull},
    {683u, 0x67ac91b2d3ba84baull}, {680u, 0x68cd100893e9e323ull}, {676u, 0x6a4fb4f22b678dbdull}, {673u, 0x6b7331bf7daa0437ull},
    {669u, 0x6cf9df411b5c9da8ull}, {666u, 0x6e206a9966f24d2aull}, {662u, 0x6fab36789c6b4537ull}, {659u, 0x70d4e0f22142bcb7ull},
    {656u, 0x71ffe71d15532491ull}, {653u, 0x732c4c2973aebefbull}, {649u, 0x74befa4c80d31c15ull}, {646u, 0x75ee9eb679f67eeaull},
    {643u, 0x771facf46467ac1cull}, {640u, 0x785228689c9b3653ull}, {637u, 0x79861481b545b657ull}, {634u, 0x7abb74bab26430cfull},
    {631u, 0x7bf24c9b45aae2a1ull}, {628u, 0x7d2a9fb80c64b379ull}, {625u, 0x7e6471b2cecde5f6ull}, {622u, 0x7f9fc63ac0f4f857ull},
    {619u, 0x80dca10cc52d0757ull}, {616u, 0x821b05f3b01d6774ull}, {613u, 0x835af8c88e7a8f47ull}, {610u, 0x849c7d72ec74d7eeull},
    {607u, 0x85df97e91eea0740ull}, {605u, 0x86b7e24f8b749c17ull}, {602u, 0x87fdaa109d23aef7ull}, {599u, 0x89451278ecd7f9cfull},
    {596u, 0x8a8e1fb794b09134ull}, {594u, 0x8b6a69c608cfd3afull}, {591u, 0x8cb63de258f9d626ull}, {588u, 0x8e03c24d7300395aull},
    {586u, 0x8ee30cef034a20dbull}, {583u, 0x90336bba039bf32full}, {580u, 0x918586c5f5e4bf02ull}, {578u, 0x9267e737c06cd34aull},
    {575u, 0x93bcf0f649f65233ull}, {573u, 0x94a14a3845bb985eull}, {570u, 0x95f94fcc20e1d8a4ull}, {568u, 0x96dfaabd86fa1647ull},
    {565u, 0x983ab9a278709be8ull}, {563u, 0x99231f5ee9a74f79ull}, {561u, 0x9a0c58d42b116668ull}, {558u, 0x9b6bbf4e9a7eb5faull},
    {556u, 0x9c5710b8cbb73a43ull}, {554u, 0x9d433b392b888970ull}, {551u, 0x9ea71573dbf15ac9ull}, {549u, 0x9f956593f6b6355cull},
    {547u, 0xa084945c7ca87ba0ull}, {544u, 0xa1ecff97c91e267bull}, {542u, 0xa2de62326449d0a3ull}, {540u, 0xa3d0a93f45169a4bull},
    {538u, 0xa4c3d6706d5d83edull}, {535u, 0xa6324d7f8770ad8dull}, {533u, 0xa727c1962b06eb6full}, {531u, 0xa81e21e6c75b4020ull},
    {529u, 0xa9157039c51ebe71ull}, {527u, 0xaa0dae5cbcc048b3ull}, {525u, 0xab06de228a9e3499ull}, {523u, 0xac010163639a9787ull},
    {521u, 0xacfc19fcea147ffaull}, {519u, 0xadf829d243487034ull}, {517u, 0xaef532cc2d1a7e8dull}, {515u, 0xaff336d9144c9071ull}
};

/* log(x) for x > 1; x = 2^e m, i the first 7 bits of m's fraction:
 * log x = e log 2 - log c_i + log1p(m c_i - 1), m c_i - 1 exact in [0, 2^-6.5) */
#ifdef __CUDACC__
__device__ __forceinline__ double ip_log(double x)
#else
static inline double ip_log(double x)
#endif
{
    const ip_u64 u = ip_bits(x);
    /* below 1 + 2^-8 (and outside the range) the fixed point holds too few of
     * the result's bits */
    if (u < 0x3ff0100000000000ull || u >= 0x4ff0000000000000ull) return log(x);
    const uint32_t e = (uint32_t)(u >> 52) - 1023u;
    const uint32_t i = (uint32_t)(u >> 45) & 0x7fu;
    const ip_log_entry t = ip_log_table[i];
    /* m c_i - 1 in units of 2^-70: the whole part leaves at the top */
    const ip_u64 rho = (((u & IP_FRACTION) | IP_IMPLICIT) * t.c) << 8;
    const uint32_t rh = (uint32_t)(rho >> 32);
    /* 1/2 - r/3 + ... - r^7/9 in units of 2^-32, then of 2^-64 */
    uint32_t p = 0x1c71c71cu;                          /* 1/9 */
    p = 0x20000000u - (ip_mulhi32(rh, p) >> 6);        /* 1/8 */
    p = 0x24924925u - (ip_mulhi32(rh, p) >> 6);        /* 1/7 */
    p = 0x2aaaaaabu - (ip_mulhi32(rh, p) >> 6);        /* 1/6 */
    p = 0x33333333u - (ip_mulhi32(rh, p) >> 6);        /* 1/5 */
    ip_u64 q = 0x4000000000000000ull - (((ip_u64)rh * p) >> 6);
    q = 0x5555555555555555ull - (ip_mulhi(rho, q) >> 6);
    q = 0x8000000000000000ull - (ip_mulhi(rho, q) >> 6);
    const ip_u64 l1p = rho - ip_mulhi(rho, ip_mulhi(rho, q) >> 6);  /* log1p, units of 2^-70 */
    ip_u64 v;
    int ex;
    if ((e | i) == 0) {
        const int n = ip_clz64(l1p);
        v = l1p << n;
        ex = 1022 - 6 - n;
    } else {
        /* units of 2^-64, hi the whole part */
        const ip_u64 ln2 = 0xb17217f7d1cf79acull, add = t.l + (l1p >> 6);
        const ip_u64 lo = e * ln2 + add;
        const uint32_t hi = (uint32_t)ip_mulhi(e, ln2) + (lo < add ? 1u : 0u);
        if (hi) {
            const int n = 64 - ip_clz64(hi);
            v = ((ip_u64)hi << (64 - n)) | (lo >> n);
            ex = 1022 + n;
        } else {
            const int n = ip_clz64(lo);
            v = lo << n;
            ex = 1022 - n;
        }
    }
    return ip_pack(0, (v >> 11) + ((v >> 10) & 1), ex);
}

/* ---- sine and cosine -------------------------------------------------------
 * |x| 2/pi = k + f with k the nearest integer, f in 128-bit fixed point (2/pi to
 * 128 bits: next to a zero of the sine or the cosine f is as small as the
 * argument's last bit, and keeps 60 bits of its own there); with g = 2 f in
 * [-1, 1] and z = g^2
 *   sin(pi/4 g) / (pi/4 g) = 1 - z (q1 - z (q2 - ...)),
 *   cos(pi/4 g)           = 1 - z (c1 - z (c2 - ...)),
 * the Taylor coefficients in units of 2^-64, those below 2^-32 in 32-bit
 * products.  Within 0.52 ulp for |x| < 64; larger arguments, infinities and NaN
 * take the library's. */

/* k, the sign of f and z = (2 f)^2 from 2/pi to 64 bits (rounded: f within two
 * units of 2^-64, which the series do not notice; |f| is above 2^-62 for every
 * double of this range that is reduced, so the sign is right) */
struct ip_turn {
    ip_u64 hi, lo, z;  /* m 2/pi in units of 2^(e - 116), m 2^(e - 52) the argument */
    uint32_t k;        /* quadrant, modulo 4 */
    ip_u64 neg;        /* sign bit of f */
};

NBCS_IHD ip_turn ip_reduce(ip_u64 u)
{
    const int sh = 1075 - ip_exponent(u);  /* 52 - e, in [47, 79] */
    const ip_u64 m = (u & IP_FRACTION) | IP_IMPLICIT;
    ip_turn t;
    t.hi = ip_mulhi(m, 0xa2f9836e4e44152aull);
    t.lo = m * 0xa2f9836e4e44152aull;
    const ip_u64 F = sh < 64 ? (t.hi << (64 - sh)) | (t.lo >> sh) : t.hi >> (sh - 64);
    const uint32_t I = sh < 64 ? (uint32_t)(t.hi >> sh) : 0u;
    t.neg = F & IP_SIGN;
    t.k = I + (uint32_t)(F >> 63);
    const ip_u64 a = t.neg ? 0ull - F : F, b = (a << 1) - (a >> 63);
    t.z = ip_mulhi(b, b);
    return t;
}

/* 2 |f| with 2/pi to 128 bits (the 64 bits above less 2^-128 of the constant
 * below), for an argument with k: shifted up to bit 63, *n places from units of
 * 2^-64 */
NBCS_IHD ip_u64 ip_angle(ip_u64 u, const ip_turn& t, int* n)
{
    const int sh = 1075 - ip_exponent(u);  /* in [47, 53] */
    const ip_u64 m = (u & IP_FRACTION) | IP_IMPLICIT;
    const ip_u64 low = 0ull - m * 0x03d8a82e0acb2240ull;
    const ip_u64 less = ip_mulhi(m, 0x03d8a82e0acb2240ull) + (low ? 1u : 0u);
    const ip_u64 mid = t.lo - less, hi = t.hi - (t.lo < less ? 1u : 0u);
    const ip_u64 F = (hi << (64 - sh)) | (mid >> sh), F1 = (mid << (64 - sh)) | (low >> sh);
    const ip_u64 a = t.neg ? ~F + (F1 ? 0u : 1u) : F, a1 = t.neg ? 0ull - F1 : F1;
    const int z = ip_clz64(a | 1ull);
    *n = z - 1;
    return (a << z) | ((a1 >> 1) >> (63 - z));
}

/* 1 - z (q1 - ...) in units of 2^-64, below 1 */
NBCS_IHD ip_u64 ip_sine_series(ip_u64 z)
{
    const uint32_t zh = (uint32_t)(z >> 32);
    uint32_t p = 0x00075092u - ip_mulhi32(zh, 0x0000043fu);
    p = 0x09ba38d0u - ip_mulhi32(zh, p);
    const ip_u64 p5 = 0x000000099c0b5523ull - ip_mulhi32(zh, p);
    ip_u64 r = 0x000006b1a0173cd4ull - ip_mulhi(z, p5);
    r = 0x00030d51c8e41b6dull - ip_mulhi(z, r);
    r = 0x00cfce5a015e2363ull - ip_mulhi(z, r);
    r = 0x1a51a6625307d323ull - ip_mulhi(z, r);
    r = 0ull - ip_mulhi(z, r);
    return r ? r : ~0ull;
}

NBCS_IHD ip_u64 ip_cosine_series(ip_u64 z)
{
    const uint32_t zh = (uint32_t)(z >> 32);
    uint32_t p = 0x00004832u - ip_mulhi32(zh, 0x00000025u);
    p = 0x006db894u - ip_mulhi32(zh, p);
    p = 0x7e74e28eu - ip_mulhi32(zh, p);
    const ip_u64 p5 = 0x00000069b47ca881ull - ip_mulhi32(zh, p);
    ip_u64 r = 0x00003c3ea0d12375ull - ip_mulhi(z, p5);
    r = 0x00155d3c7e3cbffaull - ip_mulhi(z, r);
    r = 0x040f07c206d6b0edull - ip_mulhi(z, r);
    r = 0x4ef4f326f9177969ull - ip_mulhi(z, r);
    r = 0ull - ip_mulhi(z, r);
    return r ? r : ~0ull;
}

/* |sin| of the reduced angle; x's own significand where there is nothing to
 * reduce, so that small arguments keep their relative accuracy */
NBCS_IHD double ip_sine_of(ip_u64 u, const ip_turn& t)
{
    ip_u64 A = ip_left(u);
    int e = ip_exponent(u);
    if (t.k) {
        int n;
        A = ip_mulhi(ip_angle(u, t, &n), 0xc90fdaa22168c235ull);  /* units of 2^(-64 - n) */
        const int up = (int)(A >> 63);
        A <<= 1 - up;
        e = 1021 - n + up;
    }
    ip_u64 q = ip_mulhi(A, ip_sine_series(t.z));
    if (!(q >> 63)) {
        q <<= 1;
        e -= 1;
    }
    return ip_pack(0, (q >> 11) + ((q >> 10) & 1), e);
}

NBCS_IHD double ip_cosine_of(const ip_turn& t)
{
    const ip_u64 q = ip_cosine_series(t.z);
    return ip_pack(0, (q >> 11) + ((q >> 10) & 1), 1022);
}

/* 2^-27 <= |x| < 64; below, sin x = x and cos x = 1 to half an ulp */
NBCS_IHD bool ip_turns(ip_u64 u)
{
    return ((uint32_t)(u >> 32) & 0x7fffffffu) - 0x3e400000u < 0x40500000u - 0x3e400000u;
}
NBCS_IHD bool ip_tiny(ip_u64 u) { return ((uint32_t)(u >> 32) & 0x7fffffffu) < 0x3e400000u; }

NBCS_IHD void ip_sincos(double x, double* s, double* c)
{
    const ip_u64 u = ip_bits(x);
    if (!ip_turns(u)) {
        if (ip_tiny(u)) {
            *s = x;
            *c = 1.0;
        } else {
            *s = sin(x);
            *c = cos(x);
        }
        return;
    }
    const ip_turn t = ip_reduce(u & ~IP_SIGN);
    const ip_u64 sn = ip_bits(ip_sine_of(u, t)), cs = ip_bits(ip_cosine_of(t));
    const bool odd = t.k & 1;
    /* quadrants 0 .. 3: (s, c) = (sn, cs), (cs, -sn), (-sn, -cs), (-cs, sn), sn
     * with the sign of f */
    const ip_u64 half = (t.k & 2) ? IP_SIGN : 0, next = ((t.k + 1) & 2) ? IP_SIGN : 0;
    *s = ip_double((odd ? cs : sn ^ t.neg) ^ half ^ (u & IP_SIGN));
    *c = ip_double((odd ? sn ^ t.neg : cs) ^ next);
}

NBCS_IHD double ip_sin(double x)
{
    const ip_u64 u = ip_bits(x);
    if (!ip_turns(u)) return ip_tiny(u) ? x : sin(x);
    const ip_turn t = ip_reduce(u & ~IP_SIGN);
    const ip_u64 r = (t.k & 1) ? ip_bits(ip_cosine_of(t)) : ip_bits(ip_sine_of(u, t)) ^ t.neg;
    return ip_double(r ^ ((t.k & 2) ? IP_SIGN : 0) ^ (u & IP_SIGN));
}

#endif /* NBCS_INTFP64_H */
