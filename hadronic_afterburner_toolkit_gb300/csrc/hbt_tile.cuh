// Screened pair binning of one tile pair (device code shared by the grid
// kernels of hbt_fast.cu and the persistent batch kernels of
// hbt_persist.cuh).
//
// GB300 runs FP64 at 1/58 of its FP32 rate, so every pair is first screened
// in FP32 and only the pairs that are binned pay for more work:
//
//  A. Screen (hbt_screen.cuh, every pair): certainly outside the window, its
//     q bin certain, or undecided.  Pairs not outside go to a per-warp queue.
//  B. Slot (32 queued pairs, all lanes active): the K_T and K_phi bins in
//     FP32 with error bounds (slot_of).
//  C. Histogram update.  Mixed pairs add 1 to their denominator bin.
//     Same-event pairs add q_out, q_side, q_long and cos(q.dx / hbarC):
//       FP64 form  - differences, sums and the phase q.dx exactly from
//                    fixed-point columns (hbt_fixed.cuh, values_fixed), the
//                    cos of its remainder to a table point in FP64; q_out,
//                    q_side, q_long from algebraically identical expressions
//                    (q_out = (q_x S_x + q_y S_y) / |S|, ...) in double-float
//                    on the FP32 pipe; pairs of particles outside the
//                    columns' range in FP64 (far_values), 32 at a time;
//       FP32W form - each FP64 column split once per particle into hi + lo
//                    FP32 parts; differences and the phase in double-float
//                    arithmetic on the FP32 pipe, q values in FP32, cos by
//                    quadrant reduction and FP32 Taylor polynomials
//                    (values32_split); added with one float4 vector atomic
//                    into FP32 partial bins (two arrays, even and odd warps:
//                    partials_of) that are merged into the FP64 bins with
//                    Kahan compensation.
//       The double-float form runs the FP64 form's kernels, which are faster
//       than double-float values were and more precise.
//     In the FP32-weight form a pair is evaluated as stored (i, j) and
//     oriented afterwards: swapping first and second negates every momentum
//     and position difference, so it negates q_out, q_side, q_long exactly
//     (IEEE rounding is symmetric in sign) and leaves the phase and its cos
//     unchanged.
//  D. Pairs left undecided by A or B go to another per-warp queue; the
//     reference chain runs on them 32 at a time.
//
// With q_inv histograms the same screen decides the q_inv bin too
// (screen_qinv) and a pair stays when it is inside either window.
//
// Measured on the central group (150k pions, 5.4e9 pairs in the kept tile
// pairs, 1.94e9 binned), the same-event kernel: FP64 form 121.7 -> 49.7 ms,
// FP32-weight form 94.0 -> 46.2 ms, against a scalar prefilter, a queue, a
// scalar window test with per-component bounds and, in the FP64 form, FP64
// values.  The FP64 form now keeps the shared-memory and atomics pipe 70 %,
// the issue slots 70 % and the FP64 pipe 59 % busy.
#pragma once

#include <type_traits>

#include "hbt_chain.cuh"
#include "hbt_fixed.cuh"
#include "hbt_math.cuh"
#include "hbt_screen.cuh"

namespace hbt {
namespace tile {

using namespace chain;

constexpr float U = 5.9604645e-8f;  // 2^-24
constexpr int QCAP = 64;            // per-warp compaction queue

// Summed values of the FP32-weight form.  The momentum sums and differences
// are taken in FP64 (no cancellation), then q_out, q_side, q_long follow in
// FP32 (relative error a few 1e-7).  cos: the phase is computed and reduced
// to [-pi, pi] in FP64 (Cody-Waite with a two-part 2 pi), then to
// [-pi/4, pi/4] by quadrant in FP32, where Taylor polynomials of cos (to
// x^8) and sin (to x^9) are accurate to 3e-8 and 2e-9: error < 2e-7.
template <bool BOOST>
__device__ __forceinline__ float4 values32(const Grid &g, const double *a, const double *b) {
    const double dx = a[0] - b[0], dy = a[1] - b[1];
    const double dz = a[2] - b[2], dE = a[3] - b[3];
    const float fsx = (float)(a[0] + b[0]), fsy = (float)(a[1] + b[1]);
    const float fdx = (float)dx, fdy = (float)dy, fdz = (float)dz;
    const float inv = rsqrtf(__fmaf_rn(fsx, fsx, fsy * fsy));
    float4 v;
    v.x = __fmaf_rn(fdx, fsx, fdy * fsy) * inv;
    v.y = __fmaf_rn(fdy, fsx, -(fdx * fsy)) * inv;
    if (BOOST) {
        const float sE = (float)(a[3] + b[3]), sz = (float)(a[2] + b[2]), fdE = (float)dE;
        v.z = __fmaf_rn(sE, fdz, -(sz * fdE)) * rsqrtf((sE - sz) * (sE + sz));
    } else {
        v.z = fdz;
    }
    const double ph = g.hbarC_inv * (dE * (a[7] - b[7]) - dx * (a[4] - b[4]) -
                                     dy * (a[5] - b[5]) - dz * (a[6] - b[6]));
    const double k = rint(ph * 0.15915494309189535);  // 1 / (2 pi)
    double r = __fma_rn(-k, 6.283185307179586, ph);   // 2 pi, leading double
    r = __fma_rn(-k, 2.4492935982947064e-16, r);      // 2 pi - leading double
    const float rf = (float)r;
    const float j = rintf(rf * 0.63661977f);           // 2 / pi
    float x = __fmaf_rn(-j, 1.5707963f, rf);           // pi/2 = 1.5707963 + 4.37114e-8
    x = __fmaf_rn(-j, -4.37113883e-8f, x);
    const float x2 = x * x;
    const float c = __fmaf_rn(x2, __fmaf_rn(x2, __fmaf_rn(x2, __fmaf_rn(x2, 2.48015873e-5f,
                                                                      -1.38888889e-3f),
                                                          4.16666667e-2f),
                                            -0.5f),
                              1.0f);
    const float s = x * __fmaf_rn(x2, __fmaf_rn(x2, __fmaf_rn(x2, __fmaf_rn(x2, 2.75573192e-6f,
                                                                          -1.98412698e-4f),
                                                              8.33333333e-3f),
                                                -1.66666667e-1f),
                                  1.0f);
    const int quad = ((int)j) & 3;  // cos(x + j pi/2)
    v.w = quad == 0 ? c : quad == 1 ? -s : quad == 2 ? -c : s;
    return v;
}

// ---- double-float arithmetic (value = hi + lo, two FP32 numbers) on the
// FP32 pipe, for the FP32-weight form's per-pair values.  The error-free
// transformations are Knuth's two-sum and the FMA two-product (as in
// Dekker's and Shewchuk's double-length arithmetic).
struct FF {
    float h, l;
};

__device__ __forceinline__ FF two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    const float e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return FF{s, e};
}

// a + b with |a| >= |b| (or a == 0).
__device__ __forceinline__ FF fast_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    return FF{s, __fsub_rn(b, __fsub_rn(s, a))};
}

// (ah + al) - (bh + bl) of two split FP64 values.  A split holds its value
// to 2^-48 relative; the high parts' difference is exact (two-sum) and the
// low parts add one FP32 rounding of a term below 2^-47 of the inputs.
__device__ __forceinline__ FF ff_diff(float2 a, float2 b) {
    const FF s = two_sum(a.x, -b.x);
    return two_sum(s.h, __fadd_rn(s.l, __fsub_rn(a.y, b.y)));
}

__device__ __forceinline__ FF ff_mul(FF a, FF b) {
    const float p = __fmul_rn(a.h, b.h);
    float e = __fmaf_rn(a.h, b.h, -p);
    e = __fmaf_rn(a.h, b.l, e);
    e = __fmaf_rn(a.l, b.h, e);
    return fast_two_sum(p, e);
}

__device__ __forceinline__ FF ff_add(FF a, FF b) {
    const FF s = two_sum(a.h, b.h);
    return two_sum(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}

__device__ __forceinline__ FF ff_neg(FF a) { return FF{-a.h, -a.l}; }

// Splits an FP64 value into hi = nearest FP32 and lo = nearest FP32 to the
// rest (done once per particle and tile).
__device__ __forceinline__ float2 split(double x) {
    const float h = (float)x;
    return make_float2(h, (float)(x - (double)h));
}

// The eight columns of a particle split, two to an entry of the fixed-point
// columns' arrays, and back.
__device__ __forceinline__ FixedCols split_cols(const double *v) {
    FixedCols r;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float2 a = split(v[2 * k]), b = split(v[2 * k + 1]);
        r.c[k] = make_int4(__float_as_int(a.x), __float_as_int(a.y), __float_as_int(b.x),
                           __float_as_int(b.y));
    }
    return r;
}
__device__ __forceinline__ void columns_of(const FixedCols &r, float2 *c) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
        c[2 * k] = make_float2(__int_as_float(r.c[k].x), __int_as_float(r.c[k].y));
        c[2 * k + 1] = make_float2(__int_as_float(r.c[k].z), __int_as_float(r.c[k].w));
    }
}

// x as hi + lo, two FP32 values formed from its bits on the integer pipe:
// hi is x with the significand truncated to 24 bits, lo the remaining 29
// bits truncated to 24, so that |x - hi - lo| < 2^-46 |x| (both parts carry
// the sign of x).  For x = 0 or 2^-100 <= |x| < 2^100 (momenta, their sums
// and differences); a lo part below the FP32 normal range (2^-126) is
// dropped, and magnitudes outside the range give zero.
__device__ __forceinline__ FF f64_to_ff_bits(double x) {
    const unsigned hw = (unsigned)__double2hiint(x), lw = (unsigned)__double2loint(x);
    const unsigned sign = hw & 0x80000000u, ae = hw & 0x7fffffffu;
    const bool in_range = ae - ((1023u - 100u) << 20) < (200u << 20);
    // hi: the exponent rebiased by 1023 - 127 = 896, the top 23 explicit bits
    const unsigned hb = __funnelshift_l(lw, ae - (896u << 20), 3) | sign;
    // lo: the low 29 bits r, worth r 2^(E - 1075); its leading bit is bit
    // 31 - clz(r), so the FP32 exponent field is E - 917 - clz(r)
    const unsigned r = lw & 0x1fffffffu;
    const int lz = __clz(r);
    const int e = (int)(ae >> 20) - 917 - lz;
    const unsigned lb = (r != 0u && e > 0)
                            ? ((unsigned)e << 23) | (((r << (lz & 31)) >> 8) & 0x7fffffu) | sign
                            : sign;
    return in_range ? FF{__uint_as_float(hb), __uint_as_float(lb)} : FF{0.0f, 0.0f};
}

// Limbs (h, l) of a difference or sum as a double-float in units of h: h in
// two exact conversions, l below, normalised (of a small h, l is not below
// the last bit, and ff_mul drops the product of the low parts).  The second
// for an h in [0, 2^32).
__device__ __forceinline__ FF limbs_ff(int h, int l) {
    const float f = __int2float_rn(h);
    const float r = __int2float_rn(h - __float2int_rn(f));
    return fast_two_sum(f, __fmaf_rn(__int2float_rn(l), 0x1p-30f, r));
}
__device__ __forceinline__ FF limbs_ff(unsigned h, int l) {
    const float f = __uint2float_rn(h);
    const float r = __int2float_rn((int)(h - __float2uint_rn(f)));
    return fast_two_sum(f, __fmaf_rn(__int2float_rn(l), 0x1p-30f, r));
}

// a b + c d: the two products and their sum error-free, the terms below in
// FP32, normalised.
__device__ __forceinline__ FF ff_dot(FF a, FF b, FF c, FF d) {
    const float p = __fmul_rn(a.h, b.h), q = __fmul_rn(c.h, d.h);
    float e = __fmaf_rn(a.h, b.h, -p), f = __fmaf_rn(c.h, d.h, -q);
    e = __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, e));
    f = __fmaf_rn(c.l, d.h, __fmaf_rn(c.h, d.l, f));
    const FF s = two_sum(p, q);
    return fast_two_sum(s.h, __fadd_rn(s.l, __fadd_rn(e, f)));
}

// 1 / sqrt(x): with y0 the hardware estimate and x y0^2 = 1 + e formed to
// 2^-46, y0 (1 - e / 2 + 3 e^2 / 8), the correction left as the low part.
__device__ __forceinline__ FF ff_rsqrt_fast(FF x) {
    const float y = rsqrt_approx(x.h);
    const float p = __fmul_rn(y, y), ep = __fmaf_rn(y, y, -p);
    const float e = __fmaf_rn(x.h, ep, __fmaf_rn(x.l, p, __fmaf_rn(x.h, p, -1.0f)));
    return FF{y, __fmul_rn(y, __fmul_rn(e, __fmaf_rn(0.375f, e, -0.5f)))};
}

// hi + lo rounded to FP64, its sign changed by `neg` (a sign bit), times
// 2^shift: both parts converted on the integer pipe (a zero part becomes a
// number below 1e-38, far under the rounding of any sum it enters) and added
// in FP64.
__device__ __forceinline__ double ff_scaled(FF a, unsigned neg, int shift) {
    auto conv = [&](float x) {
        const unsigned u = __float_as_uint(x) ^ neg;
        return __hiloint2double((((int)u >> 3) & (int)0x8fffffff) + ((896 + shift) << 20),
                                (int)(u << 29));
    };
    return conv(a.h) + conv(a.l);
}

// q_out, q_side and q_long of a pair from its fixed-point momenta (hbt_fixed.cuh):
// the columns (p_x, p_y) and (m, p) of both particles, the limbs h, l of their
// differences, the results' sign.  The differences and sums are exact, the rest
// in double-float (about 1e-14 relative).
template <bool BOOST>
__device__ __forceinline__ void lcms_fixed(const int4 *a, const int4 *b, const int *h,
                                           const int *l, unsigned neg, double &qo, double &qs,
                                           double &ql) {
    const FF dx = limbs_ff(h[0], l[0]), dy = limbs_ff(h[1], l[1]);
    const FF sx = limbs_ff(a[0].x + b[0].x, a[0].y + b[0].y);
    const FF sy = limbs_ff(a[0].z + b[0].z, a[0].w + b[0].w);
    const FF inv = ff_rsqrt_fast(ff_dot(sx, sx, sy, sy));
    qo = ff_scaled(ff_mul(ff_dot(dx, sx, dy, sy), inv), neg, -26);
    qs = ff_scaled(ff_mul(ff_dot(dy, sx, ff_neg(dx), sy), inv), neg, -26);
    const FF dm = limbs_ff(h[2], l[2]), dp = limbs_ff(h[3], l[3]);
    if (BOOST) {
        const FF sm = limbs_ff((unsigned)a[1].x + (unsigned)b[1].x, a[1].y + b[1].y);
        const FF sp = limbs_ff((unsigned)a[1].z + (unsigned)b[1].z, a[1].w + b[1].w);
        const FF n = ff_dot(sm, dp, ff_neg(sp), dm);
        ql = ff_scaled(ff_mul(n, ff_rsqrt_fast(ff_mul(sm, sp))), neg, -27);
    } else {
        ql = ff_scaled(ff_add(dp, ff_neg(dm)), neg, -27);
    }
}

// The limbs of the differences of a pair's columns [0, N).
template <int N>
__device__ __forceinline__ void limb_differences(const int4 *a, const int4 *b, int *h, int *l) {
#pragma unroll
    for (int k = 0; k < N; k++) {
        h[2 * k] = a[k].x - b[k].x;
        l[2 * k] = a[k].y - b[k].y;
        h[2 * k + 1] = a[k].z - b[k].z;
        l[2 * k + 1] = a[k].w - b[k].w;
    }
}

// Summed values of an accepted same-event pair from its fixed-point columns, a
// from the i-tile, b from the j-tile, negated in q when `swap` (b is the pair's
// first particle).  The phase is summed from 32 x 32 bit products: with the
// limbs (h, l) of a difference, sum of h h' (unit 2^-37 table steps), h l' + l h'
// (2^-67) and l l' (2^-97).
template <bool BOOST>
__device__ __forceinline__ void values_fixed(const Grid &g, const double *t, const FixedCols &a,
                                             const FixedCols &b, bool swap, double &qo,
                                             double &qs, double &ql, double &w) {
    int h[8], l[8];
    limb_differences<4>(a.c, b.c, h, l);
    long long hh = 0, hl = 0, ll = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        hh += (long long)h[k] * h[k + 4];
        hl += (long long)h[k] * l[k + 4];
        hl += (long long)l[k] * h[k + 4];
        ll += (long long)l[k] * l[k + 4];
    }
    lcms_fixed<BOOST>(a.c, b.c, h, l, swap ? 0x80000000u : 0u, qo, qs, ql);
    hl += ll >> 30;
    w = cos_fixed(g, t, hh + (hl >> 30), (unsigned)hl);
}

// Summed values of an accepted same-event pair of particles outside the
// fixed-point columns' range, negated in q when `swap` (algebraically the
// reference's q_out, q_side, q_long and cos(q.dx / hbarC)).  c: the FP64 columns,
// of which the pair's rows are i and j; a, b: its fixed-point momenta, which hold
// the q values where only a position is out of range.  The phase q.dx and its
// cos (table_cos: of the unrounded product with 1 / hbarC) are FP64, and so are
// the transverse differences and sums where a momentum is out of range (one
// rounding each, so that cancelling sums stay exact to the last bits).  The q
// values, which are only summed, follow in double-float on the FP32 pipe (about
// 1e-14 relative), the boosted q_long as (s_m d_p - s_p d_m) / (2 sqrt(s_m s_p))
// of m = E - p_z, p = E + p_z: s_E d_z - s_z d_E loses digits to the pair's
// rapidity, and m_j p_i - m_i p_j, without differences of near numbers, to a small
// q_long.  The FP64 numbers are split on the integer pipe, and the q values come
// back with one addition each: 27 or 35 FP64 instructions, which bound it (60
// with sincos and the hardware's conversions: 6e7 binned pairs of particles
// spread over 1000 fm 3.9 ms, 7.6 that way; over 300 fm, where most pairs of a
// warp are of near ones, 2.6 and 8.2).  Out of line to keep its registers out of
// the pair loop.
template <bool BOOST>
__device__ __noinline__ void far_values(const Grid &g, const double *t, const double *const *c,
                                        long long i, long long j, const int4 (*a)[FT],
                                        const int4 (*b)[FT], int qi, int qj, bool swap,
                                        double &qo, double &qs, double &ql, double &w) {
    const double dx = c[0][i] - c[0][j], dy = c[1][i] - c[1][j];
    const double dz = c[2][i] - c[2][j], dE = c[3][i] - c[3][j];
    const unsigned neg = swap ? 0x80000000u : 0u;
    const int4 u[2] = {a[0][qi], a[1][qi]}, v[2] = {b[0][qj], b[1][qj]};
    if (u[1].x != kFar && v[1].x != kFar) {
        int h[4], l[4];
        limb_differences<2>(u, v, h, l);
        lcms_fixed<BOOST>(u, v, h, l, neg, qo, qs, ql);
    } else {
        const FF fx = f64_to_ff_bits(dx), fy = f64_to_ff_bits(dy);
        const FF sx = f64_to_ff_bits(c[0][i] + c[0][j]), sy = f64_to_ff_bits(c[1][i] + c[1][j]);
        const FF inv = ff_rsqrt_fast(ff_dot(sx, sx, sy, sy));
        qo = ff_scaled(ff_mul(ff_dot(fx, sx, fy, sy), inv), neg, 0);
        qs = ff_scaled(ff_mul(ff_dot(fy, sx, ff_neg(fx), sy), inv), neg, 0);
        if (BOOST) {
            const FF dm = f64_to_ff_bits(dE - dz), dp = f64_to_ff_bits(dE + dz);
            const FF sm = ff_add(f64_to_ff_bits(c[3][i] - c[2][i]), f64_to_ff_bits(c[3][j] - c[2][j]));
            const FF sp = ff_add(f64_to_ff_bits(c[3][i] + c[2][i]), f64_to_ff_bits(c[3][j] + c[2][j]));
            const FF n = ff_dot(sm, dp, ff_neg(sp), dm);
            ql = ff_scaled(ff_mul(n, ff_rsqrt_fast(ff_mul(sm, sp))), neg, -1);
        } else {
            ql = swap ? -dz : dz;
        }
    }
    // q.dx = dE dt - dx dX - dy dY - dz dZ, accumulated with fused
    // multiply-adds (one rounding per term)
    double ph = dE * (c[7][i] - c[7][j]);
    ph = __fma_rn(-dx, c[4][i] - c[4][j], ph);
    ph = __fma_rn(-dy, c[5][i] - c[5][j], ph);
    ph = __fma_rn(-dz, c[6][i] - c[6][j], ph);
    w = table_cos(t, g.cph, ph);
}

// q_inv by the reference's FP64 expression (src/HBT_correlation.cpp:334-337),
// from the FP64 columns of rows i and j: bound by its 20 FP64 instructions.  (The
// momenta from shared memory changed nothing.)  From the fixed-point columns it
// cannot have the expression's precision: in double-float 45,000 pions took 12.6
// ms in the place of 17.0, but had 6e-15 rms of relative error in the place of
// 1e-16, and their 2^-57 GeV alone are 1e-15 of a q_inv of 5 MeV.
__device__ __forceinline__ double qinv64(const double *const *c, long long i, long long j,
                                         bool swap) {
    double q[4];
#pragma unroll
    for (int f = 0; f < 4; f++) q[f] = swap ? c[f][j] - c[f][i] : c[f][i] - c[f][j];
    return sqrt(-(q[3] * q[3] - q[0] * q[0] - q[1] * q[1] - q[2] * q[2]));
}

// cos of a phase given as a double-float: reduction by quadrant with pi/2
// split into three parts (12 + 12 significant bits and the rest, so that
// j times either leading part is exact for |j| < 2^11), then the FP32
// Taylor polynomials of values32.  Absolute error below 2e-7.
__device__ __forceinline__ float ff_cos(FF ph) {
    const float j = rintf(ph.h * 0.63661977f);  // 2 / pi
    float x;
    if (fabsf(j) < 2048.0f) {
        const float t1 = __fmaf_rn(-j, 1.57080078125f, ph.h);       // exact
        const FF t2 = two_sum(t1, __fmul_rn(-j, -4.453584551811218e-06f));
        x = __fadd_rn(t2.h, __fadd_rn(t2.l, __fmaf_rn(-j, -8.705515752716053e-10f, ph.l)));
    } else {
        // never on this path (|q.dx| / hbarC is a few hundred at most)
        const double r = (double)ph.h + (double)ph.l;
        const double k = rint(r * 0.6366197723675814);
        x = (float)(r - k * 1.5707963267948966);
        return cosf(x + (float)(fmod(k, 4.0)) * 1.5707964f);
    }
    const float x2 = __fmul_rn(x, x);
    const float c = __fmaf_rn(x2, __fmaf_rn(x2, __fmaf_rn(x2, __fmaf_rn(x2, 2.48015873e-5f,
                                                                    -1.38888889e-3f),
                                                        4.16666667e-2f),
                                          -0.5f),
                              1.0f);
    const float s = x * __fmaf_rn(x2, __fmaf_rn(x2, __fmaf_rn(x2, __fmaf_rn(x2, 2.75573192e-6f,
                                                                        -1.98412698e-4f),
                                                            8.33333333e-3f),
                                              -1.66666667e-1f),
                                1.0f);
    const int quad = ((int)j) & 3;  // cos(x + j pi/2)
    return quad == 0 ? c : quad == 1 ? -s : quad == 2 ? -c : s;
}

// Summed values of the FP32-weight form from split FP64 inputs, all on the
// FP32 pipe: momentum and position differences in double-float (their
// rounding relative to the difference, not to the momenta), q_out, q_side,
// q_long in FP32 (a few 1e-7 relative), the phase (q.dx)/hbarC in
// double-float and its cos by ff_cos.  a, b: the eight split columns of the
// pair's first and second particle.
template <bool BOOST>
__device__ __forceinline__ float4 values32_split(const float2 *a, const float2 *b) {
    const FF dx = ff_diff(a[0], b[0]), dy = ff_diff(a[1], b[1]);
    const FF dz = ff_diff(a[2], b[2]), dE = ff_diff(a[3], b[3]);
    const float sx = __fadd_rn(__fadd_rn(a[0].x, b[0].x), __fadd_rn(a[0].y, b[0].y));
    const float sy = __fadd_rn(__fadd_rn(a[1].x, b[1].x), __fadd_rn(a[1].y, b[1].y));
    const float inv = rsqrtf(__fmaf_rn(sx, sx, sy * sy));
    float4 v;
    v.x = __fmaf_rn(dx.h, sx, dy.h * sy) * inv;
    v.y = __fmaf_rn(dy.h, sx, -(dx.h * sy)) * inv;
    if (BOOST) {
        const float sE = __fadd_rn(__fadd_rn(a[3].x, b[3].x), __fadd_rn(a[3].y, b[3].y));
        const float sz = __fadd_rn(__fadd_rn(a[2].x, b[2].x), __fadd_rn(a[2].y, b[2].y));
        v.z = __fmaf_rn(sE, dz.h, -(sz * dE.h)) * rsqrtf((sE - sz) * (sE + sz));
    } else {
        v.z = dz.h;
    }
    FF ph = ff_mul(dE, ff_diff(a[7], b[7]));
    ph = ff_add(ph, ff_neg(ff_mul(dx, ff_diff(a[4], b[4]))));
    ph = ff_add(ph, ff_neg(ff_mul(dy, ff_diff(a[5], b[5]))));
    ph = ff_add(ph, ff_neg(ff_mul(dz, ff_diff(a[6], b[6]))));
    constexpr double hc = 1.0 / kHbarC;  // split
    ph = ff_mul(ph, FF{(float)hc, (float)(hc - (double)(float)hc)});
    v.w = ff_cos(ph);
    return v;
}

// Shared memory of a same-event tile pair.  The i-tile's arrays hold row r at
// place (r >> 2) + 32 (r & 3): warp w screens the rows w, w + 4, ... (sorted in
// momentum space, so interleaving evens out the binned pairs between warps),
// and lane k of it finds its row, and later the rows of neighbouring queue
// entries, at consecutive places, without bank conflicts.
template <bool FAR, bool QINV>
struct __align__(16) SameSmemT {
    // fixed-point columns
    int4 xi[kFixedCols][FT];
    int4 xj[kFixedCols][FT];
    float4 ta[FT];  // the i-tile's screen terms x, y, m, p
    float2 tb[FT];  // and r2, t2
    TermsPair tj[FT / 2];
    // pairs past the screen (screen_loop): up to 31 left over and 64 of a step
    uint2 queue[FT / 32][96];
    // undecided pairs, (i, j) bits: the reference chain runs on them 32 at a
    // time (inline, a warp would run it for the one or two lanes holding one)
    unsigned queue3[FT / 32][QCAP];
    // FAR (the FP64 form without q_inv histograms): pairs of far particles
    // (far_values), x = (i, j) bits | slot << 16, y = q bin; 32 at a time, as few
    // of a list's pairs in each warp's 32 would make all warps run both kinds of
    // values
    uint2 queue4[FAR ? FT / 32 : 1][FAR ? QCAP : 1];
    // with q_inv histograms: q_inv events, x = (i, j) bits, y = bin, (z, w) = the
    // pair's cosine
    uint4 queue5[QINV ? FT / 32 : 1][QINV ? QCAP : 1];
    unsigned oi[FT], oj[FT];  // original list positions (pair orientation)
    // FP64 form: 32 pairs' sums and bins on their way out
    // (add_sums)
    double2 sums[FT / 32][2][32];
    Sums *bins[FT / 32][32];
};
template <int PREC, bool QINV>
using SameSmem = SameSmemT<PREC == 0 && !QINV, QINV>;
// Place of row r in the i-tile's arrays, and back.
__device__ __forceinline__ int place_of(int r) { return (r >> 2) | ((r & 3) << 5); }
__device__ __forceinline__ int row_at(int s) { return ((s & 31) << 2) | (s >> 5); }

// A particle list as the tile kernels read it: columns (px py pz E, and x y
// z t of same-event lists), each row's position in the caller's list
// (nullptr: the rows are in the caller's order) and, on the batched path, the
// rows' fixed-point columns and screen terms (nullptr: converted here).
struct ListRows {
    const double *const *c;
    const unsigned *orig;
    const int4 *fixed;
    const float4 *terms4;
    const float2 *terms2;
    long long stride, n;
};

// Shared memory of a mixed-event tile pair.
struct __align__(16) MixedSmem {
    float4 ta[FT];  // as in SameSmem
    float2 tb[FT];
    TermsPair tj[FT / 2];
    uint2 queue[FT / 32][96];
    unsigned queue3[FT / 32][QCAP];
};

// Appends this lane's entry to the warp queue when `take`, and runs
// `process(entry, true)` on 32 queued entries whenever 32 are waiting (all
// lanes of the warp call this in step; `count` is warp-uniform).
template <class T, class F>
__device__ __forceinline__ void enqueue(T *q, int &count, bool take, T entry, int lane,
                                        F &process) {
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if (!m) return;
    if (take) q[count + __popc(m & ((1u << lane) - 1u))] = entry;
    count += __popc(m);
    __syncwarp();
    if (count >= 32) {
        process(q[lane], true);
        __syncwarp();
        if (lane < count - 32) q[lane] = q[32 + lane];
        __syncwarp();
        count -= 32;
    }
}

// Runs `process(entry, valid)` on the entries left in the queue, all lanes
// in step (lanes beyond the count pass valid = false).
template <class T, class F>
__device__ __forceinline__ void drain(T *q, int count, int lane, F &process) {
    if (count > 0) process(q[lane < count ? lane : 0], lane < count);
    __syncwarp();
}

// Sum of x over the lanes in `peers` (the lanes of the warp holding the
// same key, from __match_any_sync), left in the group's lowest lane: a tree
// over the lanes' ranks in their group, log2(group size) shuffle rounds
// (each lane adds its next remaining peer's value, then the odd ranks drop
// out and the ranks halve).  Called by all 32 lanes.
__device__ __forceinline__ double sum_peers(unsigned peers, double x) {
    const int lane = threadIdx.x & 31;
    unsigned rest = peers & (0xfffffffeu << lane);  // peers above this lane
    int rank = __popc(peers & ((1u << lane) - 1u));
    while (__any_sync(0xffffffffu, rest != 0u)) {
        const int next = __ffs(rest);  // 1-based, 0: none left
        const double t = __shfl_sync(0xffffffffu, x, next ? next - 1 : lane);
        if (next) x += t;
        rest &= ~__ballot_sync(0xffffffffu, rank & 1);
        rank >>= 1;
    }
    return x;
}

// One q_inv histogram update per group of lanes with the same bin (`key`,
// 0xffffffff: no update): the q_inv histogram has only n_KT x qnpts bins,
// which the pairs of a warp share, so per-pair atomics would queue on a few
// addresses; the groups' updates go to the CTA's private copy (QiPart), one
// sector each.  num: add q_inv and cos (numerator, same-event) or only the
// count (denominator, mixed-event).  Called by all 32 lanes.
__device__ __forceinline__ void qinv_update(const Device &d, unsigned key, double qv, double wv,
                                            bool num) {
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int lane = threadIdx.x & 31;
    const bool leader = (peers & ((1u << lane) - 1u)) == 0u && key != 0xffffffffu;
    QiPart *p = d.h.qi_part +
                (long long)(blockIdx.x % kQiCopies) * (d.g.n_KT * d.g.qnpts) + (leader ? key : 0u);
    if (num) {
        const double sq = sum_peers(peers, qv), sw = sum_peers(peers, wv);
        if (leader) {
            atomicAdd(&p->q, sq);
            atomicAdd(&p->w, sw);
            atomicAdd(&p->n, (double)__popc(peers));
        }
    } else if (leader) {
        atomicAdd(&p->den, (double)__popc(peers));
    }
}

// A mixed-event pair the screens left undecided: the reference chain
// decides.  Out of line: it runs for a few pairs per thousand, and inlined
// its registers would crowd the screen's (the kernel spilled 420 bytes).
static __device__ __noinline__ void undecided_mixed_pair(const Device &d, const double *const *l1,
                                                         const double *const *l2, long long i,
                                                         long long j, long long n1, long long n2) {
    const Chain ch = pair_chain<true>(d.g, l1[0][i], l1[1][i], l1[2][i], l1[3][i], l2[0][j],
                                      l2[1][j], l2[2][j], l2[3][j], nullptr, nullptr);
    consume<true, MODE_FAST>(d, i, j, n2, n1, ch);
}

// A same-event pair of the FP32-weight form that the screens left
// undecided: the reference chain decides; a binned pair adds its FP32
// values to the partials.  Out of line, for the same reason.
template <bool BOOST>
__device__ __noinline__ void undecided_pair32(const Device &d, const double *A, const double *B,
                                              long long i, long long j, long long n) {
    const Chain full = pair_chain<false>(d.g, A[0], A[1], A[2], A[3], B[0], B[1], B[2], B[3],
                                         A + 4, B + 4);
    if (full.ev3 != 1) {
        consume<false, MODE_FAST>(d, i, j, n, n, full);
    } else {
        const long long at = (long long)full.slot * d.g.q3 + full.bin;
        atomicAdd(partials_of(d) + at, values32<BOOST>(d.g, A, B));
        atomicAdd(d.h.cnt + at, 1ull);
    }
}

// A same-event pair of the FP64 or double-float form that the screens left
// undecided: the reference chain decides and bins it with FP64 values.  Out
// of line, so that the chain's registers do not spill in the pair loop.
static __device__ __noinline__ void undecided_pair64(const Device &d, const double *A,
                                                     const double *B, long long i, long long j,
                                                     long long n) {
    const Chain full = pair_chain<false>(d.g, A[0], A[1], A[2], A[3], B[0], B[1], B[2], B[3],
                                         A + 4, B + 4);
    consume<false, MODE_FAST>(d, i, j, n, n, full);
}

// A pair the screens left undecided, under ordered cap admission (COUNT
// or ORDER mode): the reference chain decides; the pair is counted or
// admitted at its position in the caller's lists (row, col).  Out of line,
// like the fast-mode helpers above.
template <bool MIXED, int MODE>
__device__ __noinline__ void undecided_pair_ordered(const Device &d, const double *A,
                                                    const double *B, long long row,
                                                    long long col, long long rows,
                                                    long long cols) {
    const Chain full = pair_chain<MIXED>(d.g, A[0], A[1], A[2], A[3], B[0], B[1], B[2], B[3],
                                         MIXED ? nullptr : A + 4, MIXED ? nullptr : B + 4);
    consume<MIXED, MODE>(d, row, col, cols, rows, full);
}

// Ordered cap admission of a pair the screen decided (slot, row in the
// caller's order): COUNT adds it to its row's survivor count and returns
// false; ORDER returns true when its row lies before the slot's cut row
// (the cut row itself is admitted pair by pair by k_straddle).
template <int MODE>
__device__ __forceinline__ bool admit(const Device &d, int slot, long long row, long long rows) {
    if (MODE == MODE_FAST) return true;
    if (MODE == MODE_COUNT) {
        atomicAdd(d.caps.rowcnt + (long long)slot * rows + row, 1u);
        return false;
    }
    return row < d.caps.row_cut[slot];
}

// Screen terms of row k of a list, padding past its end.
template <bool LC>
__device__ __forceinline__ Terms load_terms(const ListRows &l, long long k, float pad) {
    if (k >= l.n) return pad_terms(pad);
    if (!l.terms4) return screen_terms<LC>(l.c[0][k], l.c[1][k], l.c[2][k], l.c[3][k]);
    const float4 a = l.terms4[k];
    const float2 b = l.terms2[k];
    return Terms{a.x, a.y, a.z, a.w, b.x, b.y};
}

// Row k's columns for the values of a form (zero past the list's end): the
// fixed-point ones, or the split ones of the FP32-weight form.
template <int PREC>
__device__ __forceinline__ FixedCols load_cols(const Grid &g, const ListRows &l, long long k) {
    FixedCols r = {};
    if (k >= l.n) return r;
    if (l.fixed) {
#pragma unroll
        for (int f = 0; f < kFixedCols; f++) r.c[f] = l.fixed[f * l.stride + k];
        return r;
    }
    double v[8];
#pragma unroll
    for (int f = 0; f < 8; f++) v[f] = l.c[f][k];
    return PREC == 1 ? split_cols(v) : fixed_cols(g, g.fixed_p, v);
}

// The pair loop: screens this lane's row against particles [jbegin, jend) of
// the j-tile (jbegin even), pairs with jj <= jmin left out, and collects the
// pairs that are not certainly outside in the warp's queue; `process(entry,
// valid)` runs on 32 of them at a time, all lanes in step.  An entry is x =
// place | particle << 8 | undecided << 16, y = q bin (place: the row's,
// place_of); with q_inv histograms x also has 3-D event << 17 | q_inv event
// << 18 | q_inv bin << 20.  ORIENT: the pair's first particle is the one with
// the smaller original position (oa, oj).
template <bool BOOST, bool ORIENT, bool QINV, class F>
__device__ __forceinline__ void screen_loop(const Screen &S, const Terms &terms,
                                            const TermsPair *tj, unsigned oa, const unsigned *oj,
                                            int jmin, int jbegin, int jend, uint2 *q,
                                            F &process) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const Row a = row_of(terms);
    const f2 plus = both(S.inv_dq);
    const int steps = (jend + 1) >> 1;
    int count = 0;
    for (int jp = jbegin >> 1;; jp++) {
        const bool last = jp >= steps;
        if (!last) {
            f2 inv_dq = plus;
            if (ORIENT) {
                const uint2 o = *reinterpret_cast<const uint2 *>(oj + 2 * jp);
                inv_dq = pack2(oa > o.x ? -S.inv_dq : S.inv_dq, oa > o.y ? -S.inv_dq : S.inv_dq);
            }
            Screened r;
            if (!screen_two<BOOST, QINV>(S, a, tj[jp], inv_dq, r)) continue;
            const int jj = 2 * jp;
            bool t0 = r.take[0], t1 = r.take[1];
            unsigned f0 = r.und[0] ? 1u << 16 : 0u, f1 = r.und[1] ? 1u << 16 : 0u;
            if (QINV) {
                f0 = ((t0 && r.und[0]) || (r.takeq[0] && r.undq[0]) ? 1u << 16 : 0u) |
                     (t0 ? 1u << 17 : 0u) | (r.takeq[0] ? 1u << 18 | r.kq[0] << 20 : 0u);
                f1 = ((t1 && r.und[1]) || (r.takeq[1] && r.undq[1]) ? 1u << 16 : 0u) |
                     (t1 ? 1u << 17 : 0u) | (r.takeq[1] ? 1u << 18 | r.kq[1] << 20 : 0u);
                t0 = t0 || r.takeq[0];
                t1 = t1 || r.takeq[1];
            }
            t0 = t0 && jj > jmin;
            t1 = t1 && jj + 1 > jmin && jj + 1 < jend;
            const unsigned m0 = __ballot_sync(0xffffffffu, t0);
            const unsigned m1 = __ballot_sync(0xffffffffu, t1);
            if (!(m0 | m1)) continue;
            const unsigned e = threadIdx.x | ((unsigned)jj << 8);
            if (t0) q[count + __popc(m0 & below)] = make_uint2(e | f0, r.bin[0]);
            count += __popc(m0);
            if (t1) q[count + __popc(m1 & below)] = make_uint2((e + 256u) | f1, r.bin[1]);
            count += __popc(m1);
            __syncwarp();
        }
        // full groups of 32 from the queue's end; at the end of the tile the
        // rest
        while (count >= (last ? 1 : 32)) {
            const int take = min(count, 32);
            count -= take;
            process(q[count + min(lane, take - 1)], lane < take);
            __syncwarp();
        }
        if (last) break;
    }
}

// Adds 32 pairs' sums to their bins (bin: nullptr, none), all lanes of the
// warp in step.  The four sums of a pair are added by four neighbouring lanes,
// so that each of the four instructions touches 8 sectors of 32 bytes: with
// each lane adding its own pair's sums one after another, every instruction
// touches 32, and the L1 pipe that splits them bounded the kernel (79 % busy;
// central group 58.5 ms, 56.6 ms with the values left out and 47.2 ms with
// the additions left out; 52.3 ms this way).
__device__ __forceinline__ void add_sums(double2 (*sums)[32], Sums **bins, Sums *bin, double qo,
                                         double qs, double ql, double w) {
    const int lane = threadIdx.x & 31, c = lane & 3;
    sums[0][lane] = make_double2(qo, qs);
    sums[1][lane] = make_double2(ql, w);
    bins[lane] = bin;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int p = 8 * r + (lane >> 2);
        Sums *b = bins[p];
        const double v = reinterpret_cast<const double *>(&sums[c >> 1][p])[c & 1];
        if (b) atomicAdd(reinterpret_cast<double *>(b) + c, v);
    }
    __syncwarp();
}

// Same-event pairs of the tiles starting at i0 and j0 (i0 <= j0) of one list
// of particles.  Every unordered pair
// is visited once (position j > i); it is oriented as the reference orients
// it, q = p_first - p_second with `first` the particle earlier in the
// caller's list.  MODE selects the admission: FAST bins
// every pair; COUNT and ORDER are the two passes of ordered cap admission,
// which see each pair at its row (the earlier of its two positions in the
// caller's list).  QINV: the pairs also go to the q_inv histograms
// (invariant_radius_flag, src/HBT_correlation.cpp:331-356).  jb, je: the part
// [jb, je) of the j-tile's rows to take (jb even).
// Called by all FT threads of the CTA; the caller syncs before reusing `sm`.
template <bool AZ, bool BOOST, int PREC, int MODE = MODE_FAST, bool QINV = false>
__device__ __forceinline__ void same_tile_pair(const Device &d, SameSmem<PREC, QINV> &sm,
                                               const double *cs, const ListRows &l,
                                               long long i0, long long j0,
                                               int jb = 0, int je = FT) {
    constexpr bool LC = BOOST || QINV;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int at_i = place_of(tid);  // this thread loads row tid of each tile
    const long long n = l.n;
    const double *const *c = l.c;
    {
        const FixedCols a = load_cols<PREC>(d.g, l, i0 + tid),
                        b = load_cols<PREC>(d.g, l, j0 + tid);
#pragma unroll
        for (int f = 0; f < kFixedCols; f++) {
            sm.xi[f][at_i] = a.c[f];
            sm.xj[f][tid] = b.c[f];
        }
    }
    sm.oi[at_i] = l.orig ? (i0 + tid < n ? l.orig[i0 + tid] : 0u) : (unsigned)(i0 + tid);
    sm.oj[tid] = l.orig ? (j0 + tid < n ? l.orig[j0 + tid] : 0u) : (unsigned)(j0 + tid);
    const Terms ti = load_terms<LC>(l, i0 + tid, -1e15f);
    sm.ta[at_i] = make_float4(ti.x, ti.y, ti.m, ti.p);
    sm.tb[at_i] = make_float2(ti.r2, ti.t2);
    put_terms(sm.tj, tid, load_terms<LC>(l, j0 + tid, 1e15f));
    __syncthreads();
    const Screen &S = d.s;
    const int il = row_at(tid);  // this lane's row, at place tid
    const int jend = (int)min((long long)je, n - j0);
    // each unordered pair once; none for rows past the list's end
    const int jmin = i0 + il >= n ? FT : (i0 == j0 ? il : -1);
    unsigned *q3 = sm.queue3[w];
    int count3 = 0;

    // pairs left undecided, 32 at a time: the reference chain decides them
    // (and may hand a K_phi edge to the host), from the FP64 columns
    auto chains = [&](unsigned e, bool valid) {
        if (!valid) return;
        const int qi = e & 0xff, qj = (e >> 8) & 0xff;
        const int ri = row_at(qi);
        const long long oa = sm.oi[qi], ob = sm.oj[qj];
        const bool swap = oa > ob;
        double A[8], B[8];  // first and second particle of the pair
#pragma unroll
        for (int f = 0; f < 8; f++) {
            const double u = c[f][i0 + ri], v = c[f][j0 + qj];
            A[f] = swap ? v : u;
            B[f] = swap ? u : v;
        }
        if (MODE != MODE_FAST || QINV) {
            const long long row = MODE == MODE_FAST ? i0 + ri : (swap ? ob : oa);
            const long long col = MODE == MODE_FAST ? j0 + qj : (swap ? oa : ob);
            undecided_pair_ordered<false, MODE>(d, A, B, row, col, n, n);
            return;
        }
        if (PREC == 1)
            undecided_pair32<BOOST>(d, A, B, i0 + ri, j0 + qj, n);
        else
            undecided_pair64(d, A, B, i0 + ri, j0 + qj, n);
    };

    // one pair with its bins decided: its values; has3: its 3-D bin's record
    // (the FP32-weight form adds it here and returns none)
    // (of far particles: far, without sums; q_inv's form takes them here)
    auto decided = [&](unsigned e, int slot, unsigned bin, bool has3, double &vo, double &vs,
                       double &vl, double &vw, bool &far) -> Sums * {
        const int qi = e & 0xff, qj = (e >> 8) & 0xff;
        const unsigned oa = sm.oi[qi], ob = sm.oj[qj];
        const bool swap = oa > ob;
        if (MODE != MODE_FAST) {
            if (!admit<MODE>(d, slot, (long long)min(oa, ob), n)) return nullptr;
        }
        const long long at = (long long)slot * d.g.q3 + bin;
        if (!QINV || has3) atomicAdd(d.h.cnt + at, 1ull);
        FixedCols a, b;
#pragma unroll
        for (int f = 0; f < kFixedCols; f++) {
            a.c[f] = sm.xi[f][qi];
            b.c[f] = sm.xj[f][qj];
        }
        if (PREC == 1) {
            // the pair as stored (i, j); swapping first and second negates
            // q_out, q_side, q_long exactly and leaves the phase unchanged
            float2 sa[8], sb[8];
            columns_of(a, sa);
            columns_of(b, sb);
            float4 v = values32_split<BOOST>(sa, sb);
            if (swap) {
                v.x = -v.x;
                v.y = -v.y;
                v.z = -v.z;
            }
            if (!QINV || has3) atomicAdd(partials_of(d) + at, v);
            if (QINV) vw = (double)v.w;
            return nullptr;
        }
        far = a.c[3].x == kFar || b.c[3].x == kFar;
        if (far) {
            if (!QINV) return nullptr;
            far_values<BOOST>(d.g, cs, c, i0 + row_at(qi), j0 + qj, sm.xi, sm.xj, qi, qj, swap, vo,
                              vs, vl, vw);
        } else
            values_fixed<BOOST>(d.g, cs, a, b, swap, vo, vs, vl, vw);
        return !QINV || has3 ? d.h.sums + at : nullptr;
    };

    // 32 decided pairs of far particles
    constexpr bool kFarQueue = PREC == 0 && !QINV && MODE != MODE_COUNT;
    uint2 *q4 = sm.queue4[kFarQueue ? w : 0];
    int count4 = 0;
    auto fars = [&](uint2 f, bool valid) {
        double vo = 0.0, vs = 0.0, vl = 0.0, vw = 0.0;
        if (valid) {
            const int qi = f.x & 0xff, qj = (f.x >> 8) & 0xff;
            far_values<BOOST>(d.g, cs, c, i0 + row_at(qi), j0 + qj, sm.xi, sm.xj, qi, qj,
                              sm.oi[qi] > sm.oj[qj], vo, vs, vl, vw);
        }
        add_sums(sm.sums[w], sm.bins[w],
                 valid ? d.h.sums + ((long long)(f.x >> 16) * d.g.q3 + f.y) : nullptr, vo, vs, vl,
                 vw);
    };

    // 32 q_inv events: half of the pairs that pass the screen have one, and
    // their FP64 instructions bind this form (45,000 pions 18.8 ms a call with
    // the events taken in place, 17.0 ms with full warps of them)
    uint4 *q5 = sm.queue5[QINV ? w : 0];
    int count5 = 0;
    auto qinvs = [&](uint4 f, bool valid) {
        const int qi = f.x & 0xff, qj = (f.x >> 8) & 0xff;
        const double vq =
            valid ? qinv64(c, i0 + row_at(qi), j0 + qj, sm.oi[qi] > sm.oj[qj]) : 0.0;
        qinv_update(d, valid ? f.y : 0xffffffffu, vq, __hiloint2double((int)f.w, (int)f.z), true);
    };

    // 32 pairs that passed the screen (all lanes of the warp in step): their
    // slot, the decided pairs' values, then the undecided ones to the last
    // queue (last, so that the chain runs with nothing of the values live)
    auto process = [&](uint2 e2, bool valid) {
        const unsigned e = e2.x & 0xffffu;
        const bool has3 = !QINV || ((e2.x >> 17) & 1u), hasq = QINV && ((e2.x >> 18) & 1u);
        int slot = -2, iK = 0;
        if (valid) {
            const int qi = e & 0xff, qj = e >> 8;
            const float4 a = sm.ta[qi];
            const TermsPair &b = sm.tj[qj >> 1];
            slot = slot_of<AZ>(S, a.x, a.y, b.x[qj & 1], b.y[qj & 1], iK);
            if (slot != -2 && (((e2.x >> 16) & 1u) || (has3 && e2.y >= S.sc_q3) ||
                               (hasq && (int)(e2.x >> 20) >= S.qnpts)))
                slot = -1;
        }
        double vo = 0.0, vs = 0.0, vl = 0.0, vw = 0.0;
        Sums *bin = nullptr;
        bool far = false;
        if (slot >= 0) bin = decided(e, slot, e2.y, has3, vo, vs, vl, vw, far);
        if (PREC != 1 && MODE != MODE_COUNT)
            add_sums(sm.sums[w], sm.bins[w], bin, vo, vs, vl, vw);
        if constexpr (QINV)
            enqueue(q5, count5, slot >= 0 && hasq,
                    make_uint4(e, (unsigned)(iK * d.g.qnpts) + (e2.x >> 20),
                               (unsigned)__double2loint(vw), (unsigned)__double2hiint(vw)),
                    lane, qinvs);
        if constexpr (kFarQueue)
            enqueue(q4, count4, far, make_uint2(e | (unsigned)slot << 16, e2.y), lane, fars);
        enqueue(q3, count3, slot == -1, e, lane, chains);
    };

    // (the orientation is by original position)
    const float4 ta = sm.ta[tid];
    const float2 tb = sm.tb[tid];
    screen_loop<BOOST, true, QINV>(S, Terms{ta.x, ta.y, ta.z, ta.w, tb.x, tb.y}, sm.tj,
                                   sm.oi[tid], sm.oj, jmin, jb, jend, sm.queue[w], process);
    if constexpr (kFarQueue) drain(q4, count4, lane, fars);
    if constexpr (QINV) drain(q5, count5, lane, qinvs);
    drain(q3, count3, lane, chains);
}

// Mixed-event pairs of the list-1 tile at i0 and the list-2 tile at j0.
// Under ordered cap admission (MODE COUNT / ORDER) a pair's row and column
// are its positions in the caller's lists.  QINV, jb, je: as for
// same_tile_pair.
template <bool AZ, bool BOOST, int MODE = MODE_FAST, bool QINV = false>
__device__ __forceinline__ void mixed_tile_pair(const Device &d, MixedSmem &sm,
                                                const ListRows &la, const ListRows &lb,
                                                long long i0, long long j0,
                                                long long row_base = 0, int jb = 0,
                                                int je = FT) {
    constexpr bool LC = BOOST || QINV;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const long long n1 = la.n, n2 = lb.n;
    const double *const *l1 = la.c, *const *l2 = lb.c;
    const unsigned *orig1 = la.orig, *orig2 = lb.orig;
    const int at_i = place_of(tid);
    const Terms ti = load_terms<LC>(la, i0 + tid, -1e15f);
    sm.ta[at_i] = make_float4(ti.x, ti.y, ti.m, ti.p);
    sm.tb[at_i] = make_float2(ti.r2, ti.t2);
    put_terms(sm.tj, tid, load_terms<LC>(lb, j0 + tid, 1e15f));
    __syncthreads();
    const Screen &S = d.s;
    const int il = row_at(tid);  // this lane's row, at place tid
    const int jend = (int)min((long long)je, n2 - j0);
    const int jmin = i0 + il >= n1 ? FT : -1;
    // ordered admission: row stride of the survivor counts and key stride of
    // the deferrals (several jobs admitted together, or this job alone)
    const long long rows = d.caps.rows_total ? d.caps.rows_total : n1;
    const long long cols = d.caps.cols_key ? d.caps.cols_key : n2;
    unsigned *q3 = sm.queue3[w];
    int count3 = 0;

    // pairs the screen left undecided, 32 at a time: the reference chain
    // decides (inline, a warp would run it for one or two lanes)
    auto chains = [&](unsigned e, bool valid) {
        if (!valid) return;
        const int qi = row_at(e & 0xff), qj = (e >> 8) & 0xff;
        if (MODE != MODE_FAST || QINV) {
            const long long row = row_base + (orig1 ? (long long)orig1[i0 + qi] : i0 + qi);
            const long long col = orig2 ? (long long)orig2[j0 + qj] : j0 + qj;
            const double A[4] = {l1[0][i0 + qi], l1[1][i0 + qi], l1[2][i0 + qi], l1[3][i0 + qi]};
            const double B[4] = {l2[0][j0 + qj], l2[1][j0 + qj], l2[2][j0 + qj], l2[3][j0 + qj]};
            undecided_pair_ordered<true, MODE>(d, A, B, row, col, rows, cols);
        } else {
            undecided_mixed_pair(d, l1, l2, i0 + qi, j0 + qj, n1, n2);
        }
    };

    // 32 pairs that passed the screen (all lanes of the warp in step)
    auto process = [&](uint2 e2, bool valid) {
        const unsigned e = e2.x & 0xffffu;
        const bool has3 = !QINV || ((e2.x >> 17) & 1u), hasq = QINV && ((e2.x >> 18) & 1u);
        int slot = -2, iK = 0;
        if (valid) {
            const int qi = row_at(e & 0xff), qj = e >> 8;
            const float4 a = sm.ta[e & 0xff];
            const TermsPair &b = sm.tj[qj >> 1];
            slot = slot_of<AZ>(S, a.x, a.y, b.x[qj & 1], b.y[qj & 1], iK);
            if (slot != -2 && (((e2.x >> 16) & 1u) || (has3 && e2.y >= S.sc_q3) ||
                               (hasq && (int)(e2.x >> 20) >= S.qnpts)))
                slot = -1;
            bool admitted = slot >= 0 && has3;
            if (MODE != MODE_FAST && admitted) {
                const long long row = row_base + (orig1 ? (long long)orig1[i0 + qi] : i0 + qi);
                admitted = admit<MODE>(d, slot, row, rows);
            }
            if (admitted) atomicAdd(d.h.den + (long long)slot * d.g.q3 + e2.y, 1ull);
        }
        if (QINV)
            qinv_update(d,
                        slot >= 0 && hasq ? (unsigned)(iK * d.g.qnpts) + (e2.x >> 20) : 0xffffffffu,
                        0.0, 0.0, false);
        enqueue(q3, count3, slot == -1, e, lane, chains);
    };

    const float4 ta = sm.ta[tid];
    const float2 tb = sm.tb[tid];
    screen_loop<BOOST, false, QINV>(S, Terms{ta.x, ta.y, ta.z, ta.w, tb.x, tb.y}, sm.tj, 0u,
                                    nullptr, jmin, jb, jend, sm.queue[w], process);
    drain(q3, count3, lane, chains);
}

}  // namespace tile
}  // namespace hbt
