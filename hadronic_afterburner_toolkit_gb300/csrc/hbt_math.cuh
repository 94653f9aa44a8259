// Table-driven FP64 elementary functions of the device code, each after
// P. T. P. Tang's table-driven method (argument reduced against a table
// point, short Taylor polynomial for the remainder, product with the
// tabulated value).  Checked against the host's libm by hbt_check_math
// (include/hbt_check.h, tests/test_math_gpu.py).
#pragma once

#include <cmath>
#include <cstring>

// Cosine table of the pair kernels: cos(2 pi k / 2048) for a quarter period, k =
// 0..512 (FP64 alone: with an FP32 copy beside each entry, the random reads took
// twice the shared-memory wavefronts).  The last entry, zero, is a number too
// small to matter whose exponent fits FP32 (cos_fixed takes FP32 values from the
// bits).  Made on the host for the batched path, by each CTA elsewhere.
constexpr int kCosEntries = 513;
static inline void cos_entries(double *t) {
    for (int k = 0; k < kCosEntries - 1; k++)
        t[k] = (double)cosl(3.14159265358979323846264338327950288L * k / 1024.0L);
    t[kCosEntries - 1] = std::ldexp(1.0, -100);
}
__device__ __forceinline__ void fill_cos_entries(double *t) {
    for (int k = threadIdx.x; k < kCosEntries; k += blockDim.x)
        t[k] = k < kCosEntries - 1 ? cospi(k / 1024.0) : 0x1p-100;
}

// Points of a period that table_cos takes from it.
constexpr int COS_POINTS = 512;

// Constants of table_cos for one scale h: it returns cos(h ph) of a phase
// ph (h = 1 / hbarC for the pair numerators, h = 1 for a plain cos), with
// the product h ph never rounded.  Filled on the host by make_cos_scale.
struct CosScale {
    double c1;       // h 512 / (2 pi): table points per unit of ph
    double s1, s2;   // (2 pi / 512) / h = s1 + s2, s1 with 26 significant bits
    double h;        // h, and the Taylor coefficients of cos(h d'), sin(h d')
    double c2, c4;   //   -h^2 / 2, h^4 / 24
    double s3, s5;   //   -h^3 / 6, h^5 / 120
    unsigned lim_hi; // high word of L, the largest power of two with L c1 < 2^27
};

// (2 pi / 512) / h is formed in double-double arithmetic (2 pi as a
// two-part constant, the division's remainder taken exactly with an FMA),
// then split into s1, its leading 26 significant bits (the low 27 bits of
// the significand cleared, so that k s1 is exact for |k| < 2^27), and the
// rest s2: s1 + s2 holds the step to about 2^-79 relative.
static inline CosScale make_cos_scale(double h) {
    CosScale k;
    const double t_hi = 6.283185307179586 / 512.0, t_lo = 2.4492935982947064e-16 / 512.0;
    const double q1 = t_hi / h;
    const double q2 = (std::fma(-q1, h, t_hi) + t_lo) / h;
    unsigned long long bits;
    std::memcpy(&bits, &q1, sizeof bits);
    bits &= ~((1ull << 27) - 1);
    std::memcpy(&k.s1, &bits, sizeof bits);
    k.s2 = (q1 - k.s1) + q2;
    k.c1 = h * (512.0 / 6.283185307179586);
    k.h = h;
    k.c2 = -0.5 * h * h;
    k.c4 = h * h * h * h / 24.0;
    k.s3 = -h * h * h / 6.0;
    k.s5 = h * h * h * h * h / 120.0;
    int m = 40;
    while (m > -40 && std::ldexp(1.0, m) * k.c1 >= 134217728.0) m--;
    k.lim_hi = (unsigned)(1023 + m) << 20;
    return k;
}

// cos(h ph), table-driven (the argument reduction of P. T. P. Tang's
// table-driven elementary functions, done on ph itself): ph = k s + d' with
// s = (2 pi / 512) / h, k the integer nearest to ph c1 (the exact product,
// rounded once by an FMA against 1.5 2^52, whose low word then holds k) and
// d' from the two-part split of s, so that d = h d' is at most pi / 512 =
// 6.2e-3 in magnitude; then
//   cos(h ph) = cos(2 pi k / 512) cos d - sin(2 pi k / 512) sin d
// with cos d to d^4 and sin d to d^5 from their Taylor series in d'
// (truncation below 1e-16 and 1e-18).  |ph| >= L (k could reach 2^27;
// never on the pair path, where |q.dx| / hbarC is a few hundred at most) and
// NaN fall back to cos(h ph).
__device__ __forceinline__ double table_cos(const double *t, const CosScale &k, double ph) {
    if (!(((unsigned)__double2hiint(ph) & 0x7fffffffu) < k.lim_hi)) return cos(k.h * ph);
    const double n = __fma_rn(ph, k.c1, 6755399441055744.0);  // 1.5 2^52
    const double kd = n - 6755399441055744.0;
    double d = __fma_rn(-kd, k.s1, ph);
    d = __fma_rn(-kd, k.s2, d);
    // point j of the quarter's table (every fourth of its entries): signs of
    // the quadrant, cos and sin swapped in odd ones
    const int j = __double2loint(n), odd = j & (COS_POINTS / 4);
    const int at = (j & (COS_POINTS / 4 - 1)) * (2048 / COS_POINTS);
    const int iu = odd ? 512 - at : at;
    const unsigned turned = (unsigned)((j + COS_POINTS / 4) & (COS_POINTS / 2)) << 23;
    const double U = t[iu], V = t[512 - iu];
    const double cj = __hiloint2double(__double2hiint(U) ^ (int)turned, __double2loint(U));
    const double sj = __hiloint2double(
        __double2hiint(V) ^ (int)(turned ^ ((unsigned)odd << 24)), __double2loint(V));
    const double d2 = d * d;
    const double cd = __fma_rn(d2, __fma_rn(d2, k.c4, k.c2), 1.0);
    const double sd = d * __fma_rn(d2, __fma_rn(d2, k.s5, k.s3), k.h);
    return __fma_rn(cj, cd, -(sj * sd));
}

// Conversions with the integer pipe: the hardware's conversions to and from
// FP64 issue on the FP64 pipe.

// (float)x, rounded to nearest even; outside FP32's normal range (and for
// values that round up out of it) the hardware's conversion.
__device__ __forceinline__ float to_float_rn(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), e = (hi >> 20) & 0x7ffu;
    if (e - 897u >= 253u) return (float)x;
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const unsigned long long r = b + 0x0fffffffull + ((b >> 29) & 1ull);
    const unsigned f = (unsigned)(r >> 29) - (896u << 23);
    return __uint_as_float((f & 0x7fffffffu) | (hi & 0x80000000u));
}

// (double)n for an integer below 2^24 in magnitude.
__device__ __forceinline__ double small_to_double(int n) {
    const unsigned f = __float_as_uint(__int2float_rn(n));
    const unsigned mag = f & 0x7fffffffu;
    const unsigned hi = mag ? (f & 0x80000000u) | ((mag >> 3) + (896u << 20)) : 0u;
    return __hiloint2double((int)hi, (int)(f << 29));
}

// Table of 2^(j / 64), j = 0..63, for table_exp, filled by each CTA that
// uses it.
constexpr int EXP_TABLE = 64;
__device__ __forceinline__ void fill_exp_table(double *t) {
    for (int k = threadIdx.x; k < EXP_TABLE; k += blockDim.x) t[k] = exp2(k / 64.0);
}

// exp(x), table-driven: n = rint(x 64 / ln 2), x = n (ln 2 / 64) + r with r
// from a two-part split of ln 2 / 64 (the leading part has 28 significant
// bits, so n times it is exact for |n| < 2^25), |r| <= ln 2 / 128 = 5.4e-3;
// with j = n mod 64 and m = floor(n / 64),
//   exp x = 2^m 2^(j / 64) (1 + r + r^2 / 2 + ... + r^5 / 120)
// (truncation below 4e-17 relative), 2^m added to the exponent field.
// Outside |x| < 700 (where 2^m could leave the normal range) it calls exp().
__device__ __forceinline__ double table_exp(const double *t, double x) {
    if (!((unsigned)(__double2hiint(x) & 0x7fffffff) < 0x4085e000u)) return exp(x);  // |x| < 700
    // rounded by an addition of 1.5 2^52, whose low word then holds n
    const int n = __double2loint(__dadd_rn(__dmul_rn(x, 92.33248261689366),  // 64 / ln 2
                                           6755399441055744.0));
    const double nd = small_to_double(n);
    double r = __fma_rn(-nd, 0x1.62e42ff000000p-7, x);         // leading part
    r = __fma_rn(-nd, -6.563929801064195e-13, r);              // ln 2 / 64 - leading part
    double p = __fma_rn(r, 1.0 / 120.0, 1.0 / 24.0);
    p = __fma_rn(p, r, 1.0 / 6.0);
    p = __fma_rn(p, r, 0.5);
    p = __fma_rn(p, r, 1.0);
    p = __fma_rn(p, r, 1.0);
    const double v = t[n & (EXP_TABLE - 1)] * p;
    return __hiloint2double(__double2hiint(v) + ((n >> 6) * (1 << 20)), __double2loint(v));
}
